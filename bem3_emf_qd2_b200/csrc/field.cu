// field.cu -- domain of a point and the electromagnetic field or the modified electromagnetic
// potentials at points off the boundary (d3qd2_src/d3qd2_field.c:10-87, 203-300,
// d3qd2_src/d3qd2_setup.c:157-238), on the device.
//
//   k_domain_id  one CTA per point: solid angles of the domains' boundary elements, summed per
//                domain in the reference's domain order (a point on a vertex or in an element's
//                plane belongs to the domain being scanned)
//   k_field_part one CTA per (point, FIELD_THREADS elements of its domain): a thread evaluates its
//                element's coefficients (field.cuh; the open region's from the tabulated remainder,
//                smooth.cuh) and the weighted sums of the boundary values (E, H: EH_s; or U: mEMP_s)
//   k_field_warp the same for few points: one CTA per (point, FIELD_EPB elements), a warp per
//                quadrature point (ewald_warp.cuh) of the open region
//   k_field_sum  one CTA per point: the CTAs' partial sums in a fixed order, then the field
//   k_memp_warp, k_memp_sum  the same for the fields from the potentials' derivatives
//
// One CTA per point, a thread per element, left all but one SM idle for one point and ran its lattice
// sums one after the other.  Measured on a B200 through bem3_ctx_field and bem3_ctx_field_memp, 384
// quads: one point of type 0 14.7 -> 0.16 ms, 441 points of type 1 61.9 -> 1.55 ms, 121 points from the
// potentials' derivatives 16.5 -> 2.6 ms.
#include "field.cuh"

struct FieldArgs {
  const double* geo;
  const double* rn;
  const int* ed;
  int MN, ps;
  const int* dlist;  // positive element ids of each domain's list, domain by domain
  const int* dsd;    // sub-domain of each of them
  int doff[BEM3_MAXDOM + 1];
  int ne[BEM3_MAXDOM];
  const int* sid[BEM3_MAXDOM];
  const double* E[BEM3_MAXDOM];
  const double* dE[BEM3_MAXDOM];
  const double* H[BEM3_MAXDOM];
  const double* dH[BEM3_MAXDOM];
  const double* U[BEM3_MAXDOM];   // [ne + 1][4][4] complex (potentials at the nodes)
  const double* dU[BEM3_MAXDOM];
  double kn[2 * BEM3_MAXDOM];
  double vk0, vk1, d1x, d1y, d2x, d2y, i_detd;
  const bem3_wave* waves;
  int nwaves;
};

#define FIELD_THREADS 128
#define TWO_PI 6.28318530717958647692

// unit-cell indices of a point (q0_domain_id_l, d3qd2_setup.c:232-238)
__device__ __forceinline__ void cell_of(const FieldArgs& A, const double* rt, int& l1, int& l2)
{
  l1 = (int)floor((rt[0] * A.d2y - rt[1] * A.d2x) * A.i_detd + 0.5);
  l2 = (int)floor(-(rt[0] * A.d1y - rt[1] * A.d1x) * A.i_detd + 0.5);
}

// One CTA per point.
#define DOMID_THREADS 128
__global__ void __launch_bounds__(DOMID_THREADS) k_domain_id(FieldArgs A, int n, const double* __restrict__ r,
                                                             int* __restrict__ did, int2* __restrict__ cell)
{
  const int p = blockIdx.x;
  __shared__ double red[DOMID_THREADS / 32];
  double rt[3] = {r[3 * p], r[3 * p + 1], r[3 * p + 2]};
  int l1 = 0, l2 = 0;
  if (A.ps) {
    cell_of(A, rt, l1, l2);
    rt[0] -= (double)l1 * A.d1x + (double)l2 * A.d2x;
    rt[1] -= (double)l1 * A.d1y + (double)l2 * A.d2y;
  }
  double og[BEM3_MAXDOM];
  for (int d = 0; d < BEM3_MAXDOM; d++) og[d] = 0.0;
  int result = -1;
  for (int d = 0; d <= A.MN; d++) {
    int hit = 0;
    for (int j = A.doff[d] + threadIdx.x; j < A.doff[d + 1]; j += DOMID_THREADS) {
      const int e = A.dlist[j];
      const int nv = (int)A.geo[(size_t)e * GEO_STRIDE + GEO_NN];
      double rv[4][3];
      for (int v = 0; v < 4; v++) {
        const int node = A.ed[4 * e + v];
        for (int k = 0; k < 3; k++) rv[v][k] = A.rn[3 * node + k] - rt[k];
      }
      int flag;
      const double om = solid_angle(nv, rv, flag);
      if (flag < 0) {
        hit = 1;
      } else {
        og[d] += om;
        og[A.dsd[j]] -= om;
      }
    }
    if (__syncthreads_or(hit)) { result = d; break; }
    double tot = warp_sum(og[d]);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = tot;
    __syncthreads();
    tot = 0.0;
    for (int w = 0; w < DOMID_THREADS / 32; w++) tot += red[w];
    __syncthreads();
    if (d == 0 && fabs(tot) < TWO_PI) { result = 0; break; }
    if (tot > TWO_PI) { result = d; break; }
  }
  if (threadIdx.x == 0) {
    did[p] = result;
    cell[p] = make_int2(l1, l2);
  }
}

template <int NV>
__device__ __forceinline__ void block_sum_n(double (*red)[FIELD_THREADS], double* v)
{
  for (int j = 0; j < NV; j++) red[j][threadIdx.x] = v[j];
  __syncthreads();
  for (int o = FIELD_THREADS / 2; o > 0; o >>= 1) {
    if (threadIdx.x < o)
      for (int j = 0; j < NV; j++) red[j][threadIdx.x] += red[j][threadIdx.x + o];
    __syncthreads();
  }
}

// Incident plane waves at a point (calc_mipw_EH, m_ipw.c:164-179), added to e, h.
__device__ __forceinline__ void add_incident(const FieldArgs& A, const double* r, cplx* e, cplx* h)
{
  for (int wv = 0; wv < A.nwaves; wv++) {
    const bem3_wave& W = A.waves[wv];
    const double te = W.ki * ((r[0] - W.f[0]) * W.sin_t * W.cos_p + (r[1] - W.f[1]) * W.sin_t * W.sin_p +
                              (r[2] - W.f[2]) * W.cos_t);
    const cplx Ee = expi(te);
    for (int i = 0; i < 3; i++) {
      e[i] += mk(W.e[2 * i], W.e[2 * i + 1]) * Ee * W.E0;
      h[i] += mk(W.h[2 * i], W.h[2 * i + 1]) * Ee * W.E0;
    }
  }
}

// Table of the smooth remainder for field points (plan nullptr: none) and the warps' sums.
struct FieldGreen {
  SmoothArgs M;  // plan, table: k_field_part
  SmoothLat W;   // split of the warps' sums: k_field_warp, k_memp_warp
};

// the point's position in its cell
__device__ __forceinline__ void field_local(const FieldArgs& A, const double* r, int2 lc, double* rt)
{
  for (int i = 0; i < 3; i++) rt[i] = r[i];
  if (A.ps) {
    rt[0] -= (double)lc.x * A.d1x + (double)lc.y * A.d2x;
    rt[1] -= (double)lc.x * A.d1y + (double)lc.y * A.d2y;
  }
}

// Adds element s (position in domain d's list) with coefficients CC to a[0..2] = E, a[3..5] = H (or
// a[0..3] = U).
template <bool POT>
__device__ __forceinline__ void field_apply(const FieldArgs& A, int d, int s, const cplx* CC, cplx* a)
{
  if (POT) {
    const double *bU = A.U[d], *bdU = A.dU[d];
    const size_t b = (size_t)(4 * (s + 1)) * 4;
    for (int nn = 0; nn < 4; nn++)
      for (int i = 0; i < 4; i++) {
        const size_t q = 2 * (b + 4 * nn + i);
        a[i] += CC[nn] * mk(bdU[q], bdU[q + 1]) - CC[nn + 4] * mk(bU[q], bU[q + 1]);
      }
    return;
  }
  const double *bE = A.E[d], *bdE = A.dE[d], *bH = A.H[d], *bdH = A.dH[d];
  const size_t b = (size_t)(4 * (s + 1)) * 3;
  for (int nn = 0; nn < 4; nn++)
    for (int i = 0; i < 3; i++) {
      const size_t q = 2 * (b + 3 * nn + i);
      const cplx vdE = mk(bdE[q], bdE[q + 1]), vE = mk(bE[q], bE[q + 1]);
      const cplx vdH = mk(bdH[q], bdH[q + 1]), vH = mk(bH[q], bH[q + 1]);
      a[i] += CC[nn] * vdE - CC[nn + 4] * vE;
      a[3 + i] += CC[nn] * vdH - CC[nn + 4] * vH;
    }
}

template <bool POT>
struct FieldNV {
  static constexpr int n = POT ? 9 : 13;  // real sums per point: U or E, H (re, im), then F
};

// Partial sums [n][gridDim.y][NV] of the elements blockIdx.y * FIELD_THREADS + threadIdx.x.
template <bool POT>
__global__ void __launch_bounds__(FIELD_THREADS, 4) k_field_part(FieldArgs A, const __grid_constant__ QPLattice L, FieldGreen Gr,
                                                                 const double* __restrict__ r, const int* __restrict__ did,
                                                                 const int2* __restrict__ cell, int type,
                                                                 double* __restrict__ part, int* status)
{
  constexpr int NV = FieldNV<POT>::n;
  const int p = blockIdx.x, d = did[p];
  const int s0 = blockIdx.y * FIELD_THREADS;
  if (d < 0 || s0 >= A.ne[d]) return;
  __shared__ double red[NV][FIELD_THREADS];
  __shared__ double rad[(SMT_LMAX + 2) * FIELD_THREADS];
  double rt[3];
  field_local(A, r + 3 * p, cell[p], rt);
  const bool per = (d == 0 && A.ps == 1);
  const cplx k = mk(A.kn[2 * d], A.kn[2 * d + 1]);
  cplx a[6];
  for (int i = 0; i < 6; i++) a[i] = mk(0, 0);
  double F = 0.0;
  const int s = s0 + threadIdx.x;
  if (s < A.ne[d]) {
    const FieldGL gl = {c_xl, c_wl, c_xh, c_wh};
    const int sd = A.sid[d][s];
    cplx CC[8];
    int st;
    if (per && Gr.M.plan) {
      const FieldTable ev = {L, *Gr.M.plan, Gr.M.tab, rad + threadIdx.x, FIELD_THREADS};
      st = type >= 2 ? field_coef_gl_table(A.geo, sd, rt, type, gl, L, ev.P, ev.tab, ev.rad, ev.st, CC, F)
                     : field_coef_by<true>(A.geo, sd, rt, type, ev, CC, F);
    } else {
      st = per ? field_coef<true>(A.geo, sd, rt, k, type, L, CC, F, &gl)
               : field_coef<false>(A.geo, sd, rt, k, type, L, CC, F, &gl);
    }
    if (st < 0) record_status(status, st);
    field_apply<POT>(A, d, s, CC, a);
  }
  double v[NV];
  for (int i = 0; i < NV - 1; i++) v[i] = (i & 1) ? a[i >> 1].im : a[i >> 1].re;
  v[NV - 1] = F;
  block_sum_n<NV>(red, v);
  if (threadIdx.x < NV) part[((size_t)p * gridDim.y + blockIdx.y) * NV + threadIdx.x] = red[threadIdx.x][0];
}

// The Green's function at r (a point of a rule, relative to the field point) by this warp; every lane
// gets the values.  Points in the field point's plane: each lane does the reference's sums.
__device__ __forceinline__ int field_warp_green(const QPLattice& L, const SmoothLat& W, const double* r, int lane, cplx& G,
                                                cplx* dG)
{
  if (field_in_plane(L, r[2])) {
    QPVal v;
    const int e = field_plain_v1(L, r, v);
    G = v.G;
    for (int i = 0; i < 3; i++) dG[i] = v.dG[i];
    return e;
  }
  EwaldVal o;
  double px, py;
  ewald_terms<false>(L, W, r, lane, 32, o, &px, &py);
  double s[8] = {o.G.re, o.G.im, o.dG[0].re, o.dG[0].im, o.dG[1].re, o.dG[1].im, o.dG[2].re, o.dG[2].im};
  warp_sum_arr<8>(s);
  o.G = mk(s[0], s[1]);
  for (int i = 0; i < 3; i++) o.dG[i] = mk(s[2 + 2 * i], s[3 + 2 * i]);
  ewald_phase<false>(L, px, py, o);
  G = o.G;
  for (int i = 0; i < 3; i++) dG[i] = o.dG[i];
  return 0;
}

#define FIELD_EPB 4
// Partial sums of the elements blockIdx.y * epb .. + epb - 1 (types 0 and 1).
template <bool POT>
__global__ void __launch_bounds__(FIELD_THREADS) k_field_warp(FieldArgs A, const __grid_constant__ QPLattice L, FieldGreen Gr,
                                                              int epb, const double* __restrict__ r,
                                                              const int* __restrict__ did, const int2* __restrict__ cell,
                                                              int type, double* __restrict__ part, int* status)
{
  constexpr int NV = FieldNV<POT>::n;
  const int p = blockIdx.x, d = did[p];
  const int s0 = blockIdx.y * epb;
  if (d < 0 || s0 >= A.ne[d]) return;
  const int ne = min(epb, A.ne[d] - s0);
  __shared__ FieldKer ker[FIELD_EPB][9];
  __shared__ double red[FIELD_EPB][NV];
  double rt[3];
  field_local(A, r + 3 * p, cell[p], rt);
  const bool per = (d == 0 && A.ps == 1);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if (per) {
    for (int it = wid; it < ne * 9; it += FIELD_THREADS / 32) {
      const int j = it / 9, i = it - 9 * j, sd = A.sid[d][s0 + j];
      if (sd < 0 || i >= field_rule_points((int)A.geo[(size_t)sd * GEO_STRIDE + GEO_NN], type)) continue;
      double vR[3], vW[3];
      field_rule_point(A.geo, sd, type, i, rt, vR, vW);
      cplx G, dG[3];
      const int st = field_warp_green(L, Gr.W, vR, lane, G, dG);
      if (lane == 0) {
        FieldKer q;
        field_kernel_geom(vR, vW, q);
        q.g = G;
        q.hn = dG[0] * vW[0] + dG[1] * vW[1] + dG[2] * vW[2];
        ker[j][i] = q;
        record_status(status, st);
      }
    }
    __syncthreads();
  }
  if ((int)threadIdx.x < ne) {
    const int s = s0 + threadIdx.x, sd = A.sid[d][s];
    cplx CC[8], a[6];
    for (int i = 0; i < 6; i++) a[i] = mk(0, 0);
    double F;
    const int st = per ? field_coef_by<true>(A.geo, sd, rt, type, FieldStored{ker[threadIdx.x]}, CC, F)
                       : field_coef_by<false>(A.geo, sd, rt, type, FieldPlain<false>{L, mk(A.kn[2 * d], A.kn[2 * d + 1])}, CC, F);
    if (st < 0) record_status(status, st);
    field_apply<POT>(A, d, s, CC, a);
    for (int i = 0; i < NV - 1; i++) red[threadIdx.x][i] = (i & 1) ? a[i >> 1].im : a[i >> 1].re;
    red[threadIdx.x][NV - 1] = F;
  }
  __syncthreads();
  if (threadIdx.x < NV) {
    double s = 0.0;
    for (int j = 0; j < ne; j++) s += red[j][threadIdx.x];
    part[((size_t)p * gridDim.y + blockIdx.y) * NV + threadIdx.x] = s;
  }
}

// POT false: E, H at the points (EH_s, EH_t, EH_i for mode 0, 1, 2; d3qd2_field.c:203-300),
// Eo and Ho [n][3] complex.  POT true: U[4] (mEMP_s, mEMP_t, mEMP_i; d3qd2_field.c:10-87), Eo
// [n][4] complex, Ho unused.  mode 2 sums nothing: the incident field (or its vector potential
// U = (E_inc, 0)) at every point, whatever its domain.  part: nb partial sums per point, of epb
// elements each.
template <bool POT>
__global__ void __launch_bounds__(FIELD_THREADS) k_field_sum(FieldArgs A, const double* __restrict__ r,
                                                             const int* __restrict__ did, const int2* __restrict__ cell,
                                                             int mode, const double* __restrict__ part, int nb, int epb,
                                                             double* __restrict__ Eo, double* __restrict__ Ho)
{
  constexpr int NO = POT ? 4 : 3;  // complex outputs per vector
  constexpr int NV = FieldNV<POT>::n;
  const int p = blockIdx.x;
  const int d = did[p];
  const double r_in[3] = {r[3 * p], r[3 * p + 1], r[3 * p + 2]};
  if (mode == 2) {
    if (threadIdx.x != 0) return;
    cplx e[3], h[3];
    for (int i = 0; i < 3; i++) { e[i] = mk(0, 0); h[i] = mk(0, 0); }
    add_incident(A, r_in, e, h);
    for (int i = 0; i < 3; i++) { Eo[2 * NO * p + 2 * i] = e[i].re; Eo[2 * NO * p + 2 * i + 1] = e[i].im; }
    if (POT) { Eo[2 * NO * p + 6] = 0.0; Eo[2 * NO * p + 7] = 0.0; }
    else for (int i = 0; i < 3; i++) { Ho[6 * p + 2 * i] = h[i].re; Ho[6 * p + 2 * i + 1] = h[i].im; }
    return;
  }
  if (d < 0) {
    if (threadIdx.x < 2 * NO) Eo[2 * NO * p + threadIdx.x] = 0.0;
    if (!POT && threadIdx.x < 6) Ho[6 * p + threadIdx.x] = 0.0;
    return;
  }
  __shared__ double red[NV][FIELD_THREADS];
  double v[NV];
  for (int i = 0; i < NV; i++) v[i] = 0.0;
  const int used = (A.ne[d] + epb - 1) / epb;
  for (int c = threadIdx.x; c < used; c += FIELD_THREADS)
    for (int i = 0; i < NV; i++) v[i] += part[((size_t)p * nb + c) * NV + i];
  block_sum_n<NV>(red, v);
  if (threadIdx.x != 0) return;
  const int2 lc = cell[p];
  const double Ft = red[NV - 1][0];
  const double sc = 1.0 / ((d == 0) ? 1.0 + Ft : Ft);
  cplx o[6];
  for (int i = 0; i < (NV - 1) / 2; i++) o[i] = mk(red[2 * i][0], red[2 * i + 1][0]) * sc;
  if (lc.x != 0 || lc.y != 0) {  // Bloch phase of the cell the point lies in
    const double arg = A.vk0 * ((double)lc.x * A.d1x + (double)lc.y * A.d2x) +
                       A.vk1 * ((double)lc.x * A.d1y + (double)lc.y * A.d2y);
    const cplx ce = expi(arg);
    for (int i = 0; i < (NV - 1) / 2; i++) o[i] = o[i] * ce;
  }
  if (mode == 1 && d == 0) {  // total field: the incident waves at the point itself
    cplx e[3], h[3];
    for (int i = 0; i < 3; i++) { e[i] = mk(0, 0); h[i] = mk(0, 0); }
    add_incident(A, r_in, e, h);
    for (int i = 0; i < 3; i++) {
      o[i] += e[i];
      if (!POT) o[3 + i] += h[i];
    }
  }
  for (int i = 0; i < NO; i++) { Eo[2 * NO * p + 2 * i] = o[i].re; Eo[2 * NO * p + 2 * i + 1] = o[i].im; }
  if (!POT)
    for (int i = 0; i < 3; i++) { Ho[6 * p + 2 * i] = o[3 + i].re; Ho[6 * p + 2 * i + 1] = o[3 + i].im; }
}

// E, H from the derivatives of the potentials (EH_mEMP_s / _t / _i for mode 0, 1, 2;
// d3qd2_field.c:89-201).  The coefficient-gradient rules (field_grad_coef) give the sums U[4], dU[3][4]
// (d/dr of U), F and dF[3] over the source elements, by one of two kernels into partial sums:
//   k_memp_warp  types 0 and 1: one CTA per (point, epb elements), a warp per quadrature point of the
//                open region (ewald_warp.cuh)
//   k_memp_part  the other rules: one CTA per (point, FIELD_THREADS elements), a thread per element
// A point whose |dF/dr_p| exceeds 10 (CBD_CDF, d3qd2_const.h:84; it lies too close to the
// boundary for these rules) gets zero fields and did = -did (-99 in the open region), as the
// reference returns.  ch = lambda0 / (2 pi i).
#define EHM_CDF 10.0
#define EHM_OPENDID 99
#define MEMP_NV 36  // U (8), dU (24), F, dF (3)

__device__ __forceinline__ void memp_apply(const FieldArgs& A, int d, int s, const cplx* CC, const cplx (*dC)[8], double f,
                                           const double* df, double* v)
{
  const double *bU = A.U[d], *bdU = A.dU[d];
  const size_t b = (size_t)(4 * (s + 1)) * 4;
  for (int nn = 0; nn < 4; nn++)
    for (int i = 0; i < 4; i++) {
      const size_t q = 2 * (b + 4 * nn + i);
      const cplx vdU = mk(bdU[q], bdU[q + 1]), vU = mk(bU[q], bU[q + 1]);
      const cplx u = CC[nn] * vdU - CC[nn + 4] * vU;
      v[2 * i] += u.re;
      v[2 * i + 1] += u.im;
      for (int c = 0; c < 3; c++) {
        const cplx du = dC[c][nn] * vdU - dC[c][nn + 4] * vU;
        v[8 + 8 * c + 2 * i] += du.re;
        v[9 + 8 * c + 2 * i] += du.im;
      }
    }
  v[32] += f;
  for (int c = 0; c < 3; c++) v[33 + c] += df[c];
}

__global__ void __launch_bounds__(FIELD_THREADS) k_memp_part(FieldArgs A, const __grid_constant__ QPLattice L,
                                                             const double* __restrict__ r, const int* __restrict__ did,
                                                             const int2* __restrict__ cell, int type,
                                                             double* __restrict__ part, int* status)
{
  const int p = blockIdx.x, d = did[p];
  const int s0 = blockIdx.y * FIELD_THREADS;
  if (d < 0 || s0 >= A.ne[d]) return;
  __shared__ double red[MEMP_NV][FIELD_THREADS];
  double rt[3];
  field_local(A, r + 3 * p, cell[p], rt);
  const bool per = (d == 0 && A.ps == 1);
  const cplx k = mk(A.kn[2 * d], A.kn[2 * d + 1]);
  const FieldGL gl = {c_xl, c_wl, c_xh, c_wh};
  double v[MEMP_NV];
  for (int i = 0; i < MEMP_NV; i++) v[i] = 0.0;
  const int s = s0 + threadIdx.x;
  if (s < A.ne[d]) {
    cplx CC[8], dC[3][8];
    double f, df[3];
    const int st = per ? field_grad_coef<true>(A.geo, A.sid[d][s], rt, k, type, L, &gl, CC, dC, f, df)
                       : field_grad_coef<false>(A.geo, A.sid[d][s], rt, k, type, L, &gl, CC, dC, f, df);
    if (st < 0) record_status(status, st);
    memp_apply(A, d, s, CC, dC, f, df, v);
  }
  block_sum_n<MEMP_NV>(red, v);
  if (threadIdx.x < MEMP_NV) part[((size_t)p * gridDim.y + blockIdx.y) * MEMP_NV + threadIdx.x] = red[threadIdx.x][0];
}

#ifndef MEMP_BLOCKS
#define MEMP_BLOCKS 4
#endif
__global__ void __launch_bounds__(FIELD_THREADS, MEMP_BLOCKS) k_memp_warp(FieldArgs A, const __grid_constant__ QPLattice L, FieldGreen Gr,
                                                             int epb, const double* __restrict__ r,
                                                             const int* __restrict__ did, const int2* __restrict__ cell,
                                                             int type, double* __restrict__ part, int* status)
{
  const int p = blockIdx.x, d = did[p];
  const int s0 = blockIdx.y * epb;
  if (d < 0 || s0 >= A.ne[d]) return;
  const int ne = min(epb, A.ne[d] - s0);
  __shared__ GradKer ker[FIELD_EPB][9];
  __shared__ double red[FIELD_EPB][MEMP_NV];
  double rt[3];
  field_local(A, r + 3 * p, cell[p], rt);
  const bool per = (d == 0 && A.ps == 1);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if (per) {
    for (int it = wid; it < ne * 9; it += FIELD_THREADS / 32) {
      const int j = it / 9, i = it - 9 * j, sd = A.sid[d][s0 + j];
      if (sd < 0 || i >= field_rule_points((int)A.geo[(size_t)sd * GEO_STRIDE + GEO_NN], type)) continue;
      double vR[3], vW[3];
      field_grad_rule_point(A.geo, sd, type, i, rt, vR, vW);
      EwaldVal o;
      double px, py;
      ewald_terms<true>(L, Gr.W, vR, lane, 32, o, &px, &py);
      double* t = reinterpret_cast<double*>(&o);  // 10 complex values
#pragma unroll
      for (int c = 0; c < 20; c++) t[c] = warp_sum(t[c]);
      if (lane == 0) {
        ewald_phase<true>(L, px, py, o);
        GradKer q;
        double aR, rdW;
        grad_kernel_geom(vR, vW, q, aR, rdW);
        grad_kernel_from(o.G, o.dG, o.d2, vW, q);
        ker[j][i] = q;
      }
    }
    __syncthreads();
  }
  if ((int)threadIdx.x < ne) {
    const int s = s0 + threadIdx.x, sd = A.sid[d][s];
    cplx CC[8], dC[3][8];
    double f, df[3], v[MEMP_NV];
    for (int i = 0; i < MEMP_NV; i++) v[i] = 0.0;
    const int st = per ? field_grad_coef_by<true>(A.geo, sd, rt, type, GradStored{ker[threadIdx.x]}, nullptr, CC, dC, f, df)
                       : field_grad_coef<false>(A.geo, sd, rt, mk(A.kn[2 * d], A.kn[2 * d + 1]), type, L, nullptr, CC, dC,
                                                f, df);
    if (st < 0) record_status(status, st);
    memp_apply(A, d, s, CC, dC, f, df, v);
    for (int i = 0; i < MEMP_NV; i++) red[threadIdx.x][i] = v[i];
  }
  __syncthreads();
  if (threadIdx.x < MEMP_NV) {
    double s = 0.0;
    for (int j = 0; j < ne; j++) s += red[j][threadIdx.x];
    part[((size_t)p * gridDim.y + blockIdx.y) * MEMP_NV + threadIdx.x] = s;
  }
}

__global__ void __launch_bounds__(FIELD_THREADS) k_memp_sum(FieldArgs A, const double* __restrict__ r, int* __restrict__ did,
                                                            const int2* __restrict__ cell, int mode, double lambda0,
                                                            const double* __restrict__ part, int nb, int epb,
                                                            double* __restrict__ Eo, double* __restrict__ Ho)
{
  const int p = blockIdx.x;
  const int d = did[p];
  const double r_in[3] = {r[3 * p], r[3 * p + 1], r[3 * p + 2]};
  if (mode == 2 || d < 0) {
    if (threadIdx.x != 0) return;
    cplx e[3], h[3];
    for (int i = 0; i < 3; i++) { e[i] = mk(0, 0); h[i] = mk(0, 0); }
    if (mode == 2) add_incident(A, r_in, e, h);
    for (int i = 0; i < 3; i++) {
      Eo[6 * p + 2 * i] = e[i].re; Eo[6 * p + 2 * i + 1] = e[i].im;
      Ho[6 * p + 2 * i] = h[i].re; Ho[6 * p + 2 * i + 1] = h[i].im;
    }
    return;
  }
  __shared__ double red[MEMP_NV][FIELD_THREADS];
  double v[MEMP_NV];
  for (int i = 0; i < MEMP_NV; i++) v[i] = 0.0;
  const int used = (A.ne[d] + epb - 1) / epb;
  for (int c = threadIdx.x; c < used; c += FIELD_THREADS)
    for (int i = 0; i < MEMP_NV; i++) v[i] += part[((size_t)p * nb + c) * MEMP_NV + i];
  block_sum_n<MEMP_NV>(red, v);
  if (threadIdx.x != 0) return;
  const int2 lc = cell[p];
  const double Ft = red[32][0], dFt[3] = {red[33][0], red[34][0], red[35][0]};
  cplx e[3], h[3];
  if (fabs(dFt[0]) > EHM_CDF || fabs(dFt[1]) > EHM_CDF || fabs(dFt[2]) > EHM_CDF) {
    for (int i = 0; i < 6; i++) { Eo[6 * p + i] = 0.0; Ho[6 * p + i] = 0.0; }
    did[p] = (d == 0) ? -EHM_OPENDID : -d;
    return;
  }
  const double iC = 1.0 / ((d == 0) ? 1.0 + Ft : Ft);
  cplx u[4], du[3][4];
  for (int i = 0; i < 4; i++) u[i] = mk(red[2 * i][0], red[2 * i + 1][0]) * iC;
  for (int c = 0; c < 3; c++)
    for (int i = 0; i < 4; i++)
      du[c][i] = (mk(red[8 + 8 * c + 2 * i][0], red[9 + 8 * c + 2 * i][0]) - u[i] * dFt[c]) * iC;
  const cplx ch = mk(0.0, -lambda0 / (2.0 * QP_PI));  // lambda0 / (2 pi i)
  for (int c = 0; c < 3; c++) e[c] = u[c] - du[c][3];
  h[0] = ch * (du[1][2] - du[2][1]);
  h[1] = ch * (du[2][0] - du[0][2]);
  h[2] = ch * (du[0][1] - du[1][0]);
  if (lc.x != 0 || lc.y != 0) {
    const double arg = A.vk0 * ((double)lc.x * A.d1x + (double)lc.y * A.d2x) +
                       A.vk1 * ((double)lc.x * A.d1y + (double)lc.y * A.d2y);
    const cplx ce = expi(arg);
    for (int i = 0; i < 3; i++) { e[i] = e[i] * ce; h[i] = h[i] * ce; }
  }
  if (mode == 1 && d == 0) {
    cplx ei[3], hi[3];
    for (int i = 0; i < 3; i++) { ei[i] = mk(0, 0); hi[i] = mk(0, 0); }
    add_incident(A, r_in, ei, hi);
    for (int i = 0; i < 3; i++) { e[i] += ei[i]; h[i] += hi[i]; }
  }
  for (int i = 0; i < 3; i++) {
    Eo[6 * p + 2 * i] = e[i].re; Eo[6 * p + 2 * i + 1] = e[i].im;
    Ho[6 * p + 2 * i] = h[i].re; Ho[6 * p + 2 * i + 1] = h[i].im;
  }
}
