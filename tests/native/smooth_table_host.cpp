// Host build of the samples of the assembly's table (csrc/smooth.cuh, csrc/assemble_smooth.cuh).
#include "smooth_host.cpp"

extern "C" {

// The real-space part of a sample at r (the block of images with signs su, sv); lat as sh_plan's.  ve: the
// split parameter.
int st_real(const double* lat, const double* r, double su, double sv, double* out, double* ve)
{
  QPLattice L;
  memset((void*)&L, 0, sizeof L);
  if (qp_lattice_init(L, lat[0], lat[1], lat[2], lat[3], lat[4], lat[5], lat[6]) != 0) return 0;
  SmoothLat S;
  smooth_lattice(L, S);
  SmoothCell c;
  memset((void*)&c, 0, sizeof c);
  c.su = su;
  c.sv = sv;
  const cplx v = smooth_real(L, S, c, r);
  out[0] = v.re; out[1] = v.im;
  *ve = S.ve;
  return S.ok;
}

}
