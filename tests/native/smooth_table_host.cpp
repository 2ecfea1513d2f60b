// Host build of the assembly's table as its kernels make it (csrc/smooth.cuh, csrc/assemble_smooth.cuh): the
// centres a pair needs are filled with the spectral samples without the wave of order (0, 0), that wave's
// differences from its value at the centre, and that value in degree 0.
#include "smooth_host.cpp"

namespace {
void table_centre(int slot)
{
  SmoothPlan& P = D.P;
  if (D.have[slot]) return;
  D.have[slot] = 1;
  SmoothCell c;
  smooth_centre(D.L, P, slot % P.N1 - P.I, slot / P.N1 % P.N2 - P.J, slot / P.N1 / P.N2, c);
  const cplx K = smooth_wave_centre(D.L, c);
  std::vector<cplx> smp(P.nth * P.nph), a(P.nth), b(P.nth);
  std::vector<double> pts(3 * P.nth * P.nph);
  for (int t = 0; t < P.nth; t++) {
    for (int q = t * P.nph; q < (t + 1) * P.nph; q++) smooth_sample_point(P, c, q, &pts[3 * q]);
    for (int i = 0; i < D.S.no1 * D.S.no2; i++) {
      double ax, ay;
      const cplx f = smooth_order<true>(D.L, D.S, D.S.o1 + i / D.S.no2, D.S.o2 + i % D.S.no2,
                                        fabs(c.cz + P.rs * P.cth[t]), &ax, &ay);
      if (f.re == 0.0 && f.im == 0.0) continue;
      for (int q = t * P.nph; q < (t + 1) * P.nph; q++) smp[q] += f * expi(ax * pts[3 * q] + ay * pts[3 * q + 1]);
    }
    for (int q = t * P.nph; q < (t + 1) * P.nph; q++)
      smp[q] += smooth_wave_diff(D.L, P, c, q, K) + smooth_real(D.L, D.S, c, &pts[3 * q]);
  }
  cplx* al = D.tab.data() + (size_t)slot * smt_ncoef(P.L);
  for (int m = 0; m <= P.L; m++) {
    for (int t = 0; t < P.nth; t++) smooth_azimuth(P, smp.data(), t, m, a[t], b[t]);
    for (int l = m; l <= P.L; l++) {
      cplx A = (m == 0 && l == 0) ? K * P.c00 : mk(0, 0), B = mk(0, 0);
      for (int t = 0; t < P.nth; t++) {
        A += a[t] * P.proj[(size_t)smt_lm(P.L, m, l) * P.nth + t];
        B += b[t] * P.proj[(size_t)smt_lm(P.L, m, l) * P.nth + t];
      }
      *al++ = A;
      if (m) *al++ = B;
    }
  }
}
}  // namespace

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

// Bound of the interior kernel's rows on element s, and the longest half of its rows at the coordinates a[n].
double st_reach(const double* geo, int s, int n, const double* a, double* longest)
{
  Elem e;
  load_elem(geo, s, e);
  *longest = 0.0;
  for (int part = 0; part < (e.nn == 3 ? 3 : 1); part++)
    for (int q = 0; q < n; q++) {
      double d2 = 0.0, z0, z1 = 0.0, n0, n1 = 1.0;
      if (e.nn == 3) regi_part(part, a[q], z0, z1, n0, n1);
      for (int i = 0; i < 3; i++) {
        const double d = e.cr[i][1] * z1 + (e.cr[i][2] + e.cr[i][3] * a[q]) * n1;
        d2 += d * d;
      }
      *longest = fmax(*longest, sqrt(d2));
    }
  return regi_reach(e);
}

// The room the host gives a domain's table (coefficients), and what the plan of the elements 1..ne of geo makes of
// `cap` coefficients: its own number, 0 when the domain is left to the point-by-point sums.
double st_capacity(const double* lat, int ne)
{
  QPLattice L;
  memset((void*)&L, 0, sizeof L);
  if (qp_lattice_init(L, lat[0], lat[1], lat[2], lat[3], lat[4], lat[5], lat[6]) != 0) return -1.0;
  SmoothLat S;
  smooth_lattice(L, S);
  return (double)smooth_capacity(L, S, ne, 4.0 * (double)ne * ne, 144.0, 0.0);
}
double st_plan_size(const double* lat, const double* geo, int ne, double cap)
{
  QPLattice L;
  memset((void*)&L, 0, sizeof L);
  if (qp_lattice_init(L, lat[0], lat[1], lat[2], lat[3], lat[4], lat[5], lat[6]) != 0) return -1.0;
  SmoothLat S;
  smooth_lattice(L, S);
  double he = 0, ra = 0, be = 0, lo[3] = {1e300, 1e300, 1e300}, hi[3] = {-1e300, -1e300, -1e300}, best = 1e300, size = 0.0;
  int tri = 0;
  for (int i = 1; i <= ne; i++) {
    Elem e;
    load_elem(geo, i, e);
    smooth_extent(L, e, &he, &ra, &be, lo, hi);
    tri |= (e.nn == 3);
  }
  const SmoothExt X = {he, hi[2] - lo[2], hi[0] - lo[0], hi[1] - lo[1], ra, be};
  for (int d = SMT_LMIN; d <= SMT_LMAX; d++) {
    SmoothGrid g;
    double c;
    smooth_choose(L, S, X, 4.0 * (double)ne * ne, 144.0, 2 * tri, (long long)cap, d, g, c);
    if (g.on && c < best) {
      best = c;
      size = (double)g.ncent * smt_ncoef(d);
    }
  }
  return size;
}

// G, grad G (8 doubles a point) by the lattice sums with the propagating orders taken first; returns the lowest
// status.
int st_sums(const double* lat, const double* r, int n, double* out)
{
  QPLattice L;
  memset((void*)&L, 0, sizeof L);
  if (qp_lattice_init(L, lat[0], lat[1], lat[2], lat[3], lat[4], lat[5], lat[6]) != 0) return -1;
  std::vector<QPProp> prop(QP_PROP_CAP);
  L.nprop = qp_prop_list(L, prop.data(), QP_PROP_CAP);
  L.prop = prop.data();
  int worst = 0;
  for (int i = 0; i < n; i++) {
    QPVal v;
    const int e = qpgf_eval<QP_V1, true>(L, r + 3 * i, v);
    if (e < worst) worst = e;
    memcpy((void*)(out + 8 * i), (const void*)&v, sizeof v);
  }
  return worst;
}

// Points per direction of the smooth rule.
int st_nq(double k, double h, double d, double bend, int tri) { return smooth_nq(k, h, d, bend, tri); }

// sh_pair by the table as the kernels make it.
int st_pair(const double* geo, int t, int tn, int s, int n, const double* x, const double* w, double* out)
{
  Elem es;
  load_elem(geo, s, es);
  const double* rt = geo + (size_t)t * GEO_STRIDE + GEO_REN + 3 * tn;
  const double v[3] = {es.cr[0][0] - rt[0], es.cr[1][0] - rt[1], es.cr[2][0] - rt[2]};
  double sx, sy;
  smooth_shift(D.L, v, &sx, &sy);
  const double* tq = es.nn == 4 ? D.P.q4 : D.P.q3;
  for (int q = 0; q < (es.nn == 4 ? D.P.nq4 : D.P.nq3); q++) {
    double r[3], W[3];
    point_geom(es, tq[3 * q], tq[3 * q + 1], rt, r, W);
    SmoothCell c;
    smooth_cell(D.L, D.P, r[0] + sx, r[1] + sy, fabs(r[2]), c);
    table_centre(c.slot);
  }
  int ip;
  return sh_pair(geo, t, tn, s, 0, n, x, w, out, &ip);
}

}
