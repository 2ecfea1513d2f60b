// assemble_smooth.cuh -- kernels of the periodic domain's matrices with the Green's function split
// into its nearest image and a tabulated smooth remainder (smooth.cuh).
//
//   k_smooth_plan     one CTA: extents of the elements, the cheapest degree and grid, the tables
//   k_smooth_spectral the spectral part of every sample of the remainder around the grid's centres:
//                     one CTA per layer of centres, height and group of azimuths
//   k_smooth_project  one CTA per centre: the samples' real-space part, then the coefficients
//   k_reg_smooth      regular pairs, one warp per SMT_PAIRS sources of a row
//   k_gh_smooth       near-singular pairs, one CTA each
//   k_self_smooth     self pairs, one CTA each
//
// Measured on a B200 against one lattice sum per point (k_reg_periodic, k_gh_periodic and
// k_self_periodic, ~200 terms a point): the open region of 96 quads 41.4 -> 2.26 ms, of 864 quads
// 1,767 -> 59.6 ms, of 352 triangles 437 -> 54 ms (33 ms of it the in-plane pairs, which stay there).
// With k_reg_smooth's evaluation tuned since, 864 quads take 39.0 ms, and with eight lanes a pair and
// fewer points for distant pairs in its nearest image (rule_order) 35.1 ms; 96 quads 1.9 ms, 352 triangles 47 ms.
// k_reg_smooth has the FP64 pipe 61 % busy with 16 warps a multiprocessor, k_smooth_project 40 %, k_smooth_spectral
// 35 % (issue slots 61 %: index arithmetic of the transform).
//
// Every kernel returns at once when the plan is off (SmoothPlan::on == 0); the point-by-point kernels
// then do the domain.  Nothing is kept between calls: plan and table are made again by each assembly.
#pragma once

#include "smooth.cuh"

// Device memory of a domain's plan and table (part of the caller's scratch) and the lattice's part.
struct SmoothArgs {
  SmoothLat S;
  SmoothPlan* plan;  // nullptr: no table for this domain
  cplx* tab;         // [cap] coefficients, centre by centre
  cplx* smp;         // [2 cap] samples
  long long cap;
};

#define SMT_PLAN_THREADS 256
__device__ __forceinline__ double block_reduce(double v, double* red, bool mx)
{
  red[threadIdx.x] = v;
  __syncthreads();
  for (int o = blockDim.x / 2; o > 0; o >>= 1) {
    if ((int)threadIdx.x < o) {
      const double a = red[threadIdx.x], b = red[threadIdx.x + o];
      red[threadIdx.x] = mx ? fmax(a, b) : fmin(a, b);
    }
    __syncthreads();
  }
  const double r = red[0];
  __syncthreads();
  return r;
}

// What the table is for: the pairs of a domain, or (points) evaluations at points of heights zlo .. zhi
// against every element, `evals` of them (near = 0: each a single point; else elements with a rule of
// `near` points per quad), `chain` in turn by a thread.
struct SmoothUse {
  int points;
  double zlo, zhi, evals, near, chain;
};

__device__ __forceinline__ void smooth_plan_block(const AssembleArgs& A, const QPLattice& L, const SmoothArgs& M,
                                                  const SmoothUse U = SmoothUse{0, 0.0, 0.0, 0.0, 0.0, 0.0})
{
  __shared__ double red[SMT_PLAN_THREADS];
  __shared__ SmoothGrid best;
  __shared__ double costs[SMT_LMAX + 1];
  double he = 0.0, ra = 0.0, be = 0.0, lo[3] = {1e300, 1e300, 1e300}, hi[3] = {-1e300, -1e300, -1e300}, tri = 0.0, quad = 0.0;
  for (int i = threadIdx.x; i < A.ne; i += blockDim.x) {
    Elem e;
    load_elem(A.geo, abs(A.sid[i]), e);
    smooth_extent(L, e, &he, &ra, &be, lo, hi);
    (e.nn == 3 ? tri : quad) = 1.0;
  }
  SmoothExt X;
  X.half_edge = block_reduce(he, red, true);
  X.radius = block_reduce(ra, red, true);
  X.bend = block_reduce(be, red, true);
  tri = block_reduce(tri, red, true);
  quad = block_reduce(quad, red, true);
  const int kinds = tri > 0.0 ? (quad > 0.0 ? 1 : 2) : 0;
  for (int i = 0; i < 3; i++) {
    const double a = block_reduce(lo[i], red, false), b = block_reduce(hi[i], red, true);
    (i == 0 ? X.ulen : i == 1 ? X.vlen : X.zlen) = b - a;
    if (i == 2 && U.points) X.zlen = fmax(fmax(U.zhi - a, b - U.zlo), 0.0);
  }
  if (U.points) X.ulen = X.vlen = 1.0;  // points anywhere in the cell
  const double np = U.points ? U.evals : 4.0 * (double)A.ne * A.ne;
  const double near = U.points ? U.near : 144.0;
  const int d = SMT_LMIN + (int)threadIdx.x;
  SmoothGrid g;
  g.on = 0;
  double c = 1e300;
  if (d <= SMT_LMAX) {
    smooth_choose(L, M.S, X, np, near, kinds, M.cap, d, g, c, U.chain);
    if (!g.on) c = 1e300;
    costs[d] = c;
  }
  __syncthreads();
  if (d <= SMT_LMAX) {
    bool mine = true;
    for (int q = SMT_LMIN; q <= SMT_LMAX; q++)
      if (costs[q] < c || (costs[q] == c && q < d)) mine = false;
    if (mine && g.on) best = g;
    if (threadIdx.x == 0) {
      bool any = false;
      for (int q = SMT_LMIN; q <= SMT_LMAX; q++) any = any || costs[q] < 1e300;
      if (!any) best.on = 0;
    }
  }
  __syncthreads();
  __shared__ SmoothPlan P;
  if (threadIdx.x == 0) *static_cast<SmoothGrid*>(&P) = best;
  __syncthreads();
  if (best.on) {
    smooth_tables_a(P, threadIdx.x, blockDim.x);
    __syncthreads();
    smooth_tables_b(P, threadIdx.x, blockDim.x);
    __syncthreads();
    smooth_tables_c(P, L.k, threadIdx.x, blockDim.x);
    __syncthreads();
  }
  const size_t words = (best.on ? sizeof(SmoothPlan) : sizeof(SmoothGrid)) / sizeof(double);
  for (size_t i = threadIdx.x; i < words; i += blockDim.x) ((double*)M.plan)[i] = ((const double*)&P)[i];
}

__global__ void __launch_bounds__(SMT_PLAN_THREADS) k_smooth_plan(AssembleArgs A, const __grid_constant__ QPLattice L,
                                                                  SmoothArgs M)
{
  smooth_plan_block(A, L, M);
}

// A table for evaluations at field points.
__global__ void __launch_bounds__(SMT_PLAN_THREADS) k_field_plan(AssembleArgs A, const __grid_constant__ QPLattice L,
                                                                 SmoothArgs M, double zlo, double zhi, double evals, double near,
                                                                 double chain)
{
  smooth_plan_block(A, L, M, SmoothUse{1, zlo, zhi, evals, near, chain});
}

__device__ __forceinline__ void smooth_slot(const QPLattice& L, const SmoothPlan& P, int slot, SmoothCell& c)
{
  const int i = slot % P.N1, q = slot / P.N1, j = q % P.N2, m = q / P.N2;
  smooth_centre(L, P, i - P.I, j - P.J, m, c);
}

// Spectral part of the samples of layer m's centres at height node t and azimuths f = g, g + SMT_FG, ...:
// sum over the orders of (height function) e^{i a.(c + rho)}, rho the sample's offset, c = (i / n1) d1 +
// (j / n2) d2.  As a.c = -k||.c + 2 pi (q1 i / n1 + q2 j / n2), the sum over all centres of the layer is
// a two-dimensional Fourier sum, done over q2 and then over q1 (16 columns j at a time).
#define SMT_FG 4
#define SMT_JT 16
#define SMT_SPEC_THREADS 256
#define SMT_SPEC_SMEM (int)(sizeof(cplx) * (2 * SMT_ORDERS + 128 * SMT_JT))  // most that smooth_spec_smem gives: 188 KB
static inline size_t smooth_spec_smem(const SmoothLat& S)
{
  return sizeof(cplx) * ((size_t)2 * S.no1 * S.no2 + (size_t)S.no1 * SMT_JT);
}
__device__ __forceinline__ void smooth_spectral_block(const QPLattice& L, const SmoothArgs& M, int first, int stride,
                                                      unsigned char* spec_smem)
{
  const SmoothPlan& P = *M.plan;
  if (!P.on) return;
  const SmoothLat& S = M.S;
  const int no = S.no1 * S.no2, ns = P.nth * P.nph;
  cplx* F = (cplx*)spec_smem;  // height functions of this block's height
  cplx* T = F + no;            // times e^{i a.rho} of one azimuth
  cplx* Z = T + no;            // [no1][SMT_JT] summed over q2
  __shared__ cplx tw1[400], tw2[400];
  for (int i = threadIdx.x; i < P.n1; i += blockDim.x) tw1[i] = expi(2.0 * QP_PI * i / P.n1);
  for (int i = threadIdx.x; i < P.n2; i += blockDim.x) tw2[i] = expi(2.0 * QP_PI * i / P.n2);
  const int items = P.N3 * P.nth * SMT_FG;
  for (int it = first; it < items; it += stride) {
    const int g = it % SMT_FG, t = it / SMT_FG % P.nth, m = it / (SMT_FG * P.nth);
    const double z = fabs(m * P.hz + P.rs * P.cth[t]);
    __syncthreads();
    for (int i = threadIdx.x; i < no; i += blockDim.x) {
      double ax, ay;
      F[i] = smooth_order<true>(L, S, S.o1 + i / S.no2, S.o2 + i % S.no2, z, &ax, &ay);
    }
    for (int f = g; f < P.nph; f += SMT_FG) {
      const double rx = P.rs * P.sth[t] * P.cph[f], ry = P.rs * P.sth[t] * P.sph[f];
      __syncthreads();
      for (int i = threadIdx.x; i < no; i += blockDim.x) {
        const int q1 = S.o1 + i / S.no2, q2 = S.o2 + i % S.no2;
        const double ax = -L.vkx + (double)q1 * L.g1x + (double)q2 * L.g2x;
        const double ay = -L.vky + (double)q1 * L.g1y + (double)q2 * L.g2y;
        const cplx v = F[i];
        T[i] = (v.re != 0.0 || v.im != 0.0) ? v * expi(ax * rx + ay * ry) : v;
      }
      __syncthreads();
      for (int j0 = 0; j0 < P.N2; j0 += SMT_JT) {
        const int nj = min(SMT_JT, P.N2 - j0);
        for (int i = threadIdx.x; i < S.no1 * SMT_JT; i += blockDim.x) {
          const int a = i / SMT_JT, jj = i % SMT_JT;
          if (jj >= nj) continue;
          const int j = j0 + jj - P.J;
          const int jm = (j % P.n2 + P.n2) % P.n2;
          int q = (int)((((long long)S.o2 * jm) % P.n2 + P.n2) % P.n2);
          cplx s = mk(0.0, 0.0);
          for (int b = 0; b < S.no2; b++) {
            s += T[a * S.no2 + b] * tw2[q];
            q += jm;
            if (q >= P.n2) q -= P.n2;
          }
          Z[i] = s;
        }
        __syncthreads();
        for (int i = threadIdx.x; i < P.N1 * nj; i += blockDim.x) {
          const int ii = i / nj, jj = i - ii * nj;
          const int im = ((ii - P.I) % P.n1 + P.n1) % P.n1;
          int q = (int)((((long long)S.o1 * im) % P.n1 + P.n1) % P.n1);
          cplx s = mk(0.0, 0.0);
          for (int a = 0; a < S.no1; a++) {
            s += Z[a * SMT_JT + jj] * tw1[q];
            q += im;
            if (q >= P.n1) q -= P.n1;
          }
          const double u = (ii - P.I) * P.rn1, v = (j0 + jj - P.J) * P.rn2;
          const cplx ph = expi(-(L.vkx * (u * L.d1x + v * L.d2x) + L.vky * (u * L.d1y + v * L.d2y)));
          const long long slot = ((long long)m * P.N2 + j0 + jj) * P.N1 + ii;
          M.smp[slot * ns + t * P.nph + f] = s * ph;
        }
        __syncthreads();
      }
    }
  }
}

__global__ void __launch_bounds__(SMT_SPEC_THREADS) k_smooth_spectral(const __grid_constant__ QPLattice L, SmoothArgs M)
{
  extern __shared__ __align__(16) unsigned char spec_smem[];
  smooth_spectral_block(L, M, blockIdx.x, gridDim.x, spec_smem);
}

#define SMT_PROJ_THREADS 128
__device__ __forceinline__ void smooth_project_block(const QPLattice& L, const SmoothArgs& M, int first, int stride)
{
  const SmoothPlan& P = *M.plan;
  if (!P.on) return;
  __shared__ cplx smp[2 * (SMT_LMAX + 1) * (SMT_LMAX + 1)];
  __shared__ cplx ca[(SMT_LMAX + 1) * (SMT_LMAX + 1)], cb[(SMT_LMAX + 1) * (SMT_LMAX + 1)];
  const int ns = P.nth * P.nph, L1 = P.L + 1;
  for (int slot = first; slot < P.ncent; slot += stride) {
    const cplx* in = M.smp + (size_t)slot * ns;
    SmoothCell c;
    smooth_slot(L, P, slot, c);
    cplx K = mk(0.0, 0.0);
    if (smooth_split(L)) {
      K = smooth_wave_centre(L, c);
      for (int i = threadIdx.x; i < ns; i += blockDim.x) smp[i] = smooth_wave_diff(L, P, c, i, K);
    }
#pragma unroll 1
    for (int i = threadIdx.x; i < ns; i += blockDim.x) {
      double r[3];
      smooth_sample_point(P, c, i, r);
      const cplx v = in[i] + smooth_real(L, M.S, c, r);
      smp[i] = smooth_split(L) ? smp[i] + v : v;
    }
    __syncthreads();
    for (int i = threadIdx.x; i < P.nth * L1; i += blockDim.x) smooth_azimuth(P, smp, i / L1, i % L1, ca[i], cb[i]);
    __syncthreads();
    cplx* al = smt_at(M.tab, P.L, slot);
    for (int i = threadIdx.x; i < L1 * L1; i += blockDim.x) {
      const int m = i / L1, l = i % L1;
      if (l < m) continue;
      const int lm = smt_lm(P.L, m, l);
      const double* w = P.proj + lm * P.nth;
      cplx a = mk(0.0, 0.0), b = mk(0.0, 0.0);
      for (int t = 0; t < P.nth; t++) {
        a += ca[t * L1 + m] * w[t];
        b += cb[t * L1 + m] * w[t];
      }
      if (m == 0) {
        al[l] = l == 0 ? a + K * P.c00 : a;
      } else {  // m >= 1: A, B in turn; (m, l) of m >= 1 start at L + 1
        const int o = L1 + 2 * (lm - L1);
        al[o] = a;
        al[o + 1] = b;
      }
    }
    __syncthreads();
  }
}

__global__ void __launch_bounds__(SMT_PROJ_THREADS) k_smooth_project(const __grid_constant__ QPLattice L, SmoothArgs M)
{
  smooth_project_block(L, M, blockIdx.x, gridDim.x);
}

// ------------------------------------------------------------------------------------------
// Regular pairs.  A warp takes SMT_PAIRS consecutive sources of one row: their rule points for the
// nearest image and the solid angle (eight lanes a pair, sums in registers), then their
// smooth points, all four pairs' in one list so that few lanes idle (4 x 36 points: 4.5 of 5 passes).
// The smooth points' values go to shared memory, from where two lanes per (pair, shape function) add
// them up: no reduction over lanes.
#define SMT_PAIRS 4
#define SMT_WARPS 1
#ifndef SMT_BLOCKS
#define SMT_BLOCKS 16  // 128 registers; with 168 (12 warps) 864 quads take 35.7 ms, with 96 (20, spills) 41.7, so 31.3
#endif
#define SMT_BUF 160  // smooth points of a pass over the list
struct SmoothWarp {
  Elem es[SMT_PAIRS];
  double tot[SMT_PAIRS][19];   // nearest image: G, H (re, im), F, dF0, dF1
  cplx sm[SMT_PAIRS][4][2];    // smooth part: G, H per shape function
  double rt[3], v0[3], v1[3];
  double sx[SMT_PAIRS], sy[SMT_PAIRS];
  int sh[SMT_PAIRS], n[SMT_PAIRS];  // shifted or not; the nearest image's points per direction
  union {
    double slot[32 * 19];              // the lanes' nearest-image sums
    struct {
      cplx buf[SMT_BUF][2];            // smooth points: g w |W|, h w
      double rad[(SMT_LMAX + 2) * 32]; // f_l of the lanes' points
    };
  };
};

// Unit `unit` of the rows r0, r0 + 1, ...: sources 4 (unit mod upr) .. + 3 of row r0 + unit / upr, by one
// warp.  xr, wr: the Gauss rules of 6 to 12 points in shared memory.
__device__ __forceinline__ void reg_smooth_unit(const AssembleArgs& A, const QPLattice& L, const SmoothArgs& M, int r0,
                                                long long unit, double3* Fp, unsigned* gh_list, unsigned* gh_count,
                                                unsigned gh_cap, unsigned* ip_list, unsigned* ip_count, int* status,
                                                SmoothWarp& w, const double* xr, const double* wr, int lane)
{
  const SmoothPlan& P = *M.plan;
  const int upr = (A.ne + SMT_PAIRS - 1) / SMT_PAIRS;
  const int rr = (int)(unit / upr), s0 = (int)(unit - (long long)rr * upr) * SMT_PAIRS;
  const int row = r0 + rr, t = row >> 2, tn = row & 3;
  double rt[3], v0[3], v1[3];
  int tnn;
  target_info(A.geo, A.sid, t, tn, rt, v0, v1, tnn);
  if (tn == 3 && tnn == 3) return;
  const int np = min(SMT_PAIRS, A.ne - s0);
  for (int i = lane; i < np * 21; i += 32) {
    const int j = i / 21, c = i - 21 * j;
    const double* g = A.geo + (size_t)abs(A.sid[s0 + j]) * GEO_STRIDE;
    const bool tri = g[GEO_NN] == 3.0;
    const bool zero = tri && (c < 12 ? (c & 3) == 3 : (c - 12) % 3 != 0);
    reinterpret_cast<double*>(&w.es[j])[c] = zero ? 0.0 : g[c];
    if (c == 0) w.es[j].nn = tri ? 3 : 4;
  }
  if (lane < 3) { w.rt[lane] = rt[lane]; w.v0[lane] = v0[lane]; w.v1[lane] = v1[lane]; }
  __syncwarp();
  bool ok = false;
  if (lane < np && s0 + lane != t) {
    const Elem& e = w.es[lane];
    const double v[3] = {e.cr[0][0] - rt[0], e.cr[1][0] - rt[1], e.cr[2][0] - rt[2]};
    w.sh[lane] = smooth_shift(L, v, &w.sx[lane], &w.sy[lane]);
    ok = !smooth_in_plane(L, e, rt[2]);
    // both the nearest image and (solid angle) the element itself are at least this far
    const double x = v[0] + w.sx[lane], y = v[1] + w.sy[lane], h2 = v[0] * v[0] + v[1] * v[1];
    w.n[lane] = rule_order(e, fmin(h2, x * x + y * y) + v[2] * v[2], L.k);
    if (!ok) ip_list[atomicAdd(ip_count, 1u)] = (unsigned)((long long)rr * A.ne + s0 + lane);
  }
  const unsigned valid = __ballot_sync(0xffffffffu, ok);
  if (valid == 0) return;
  __syncwarp();
  // nearest image: eight lanes a pair, over its 36 to 144 points (three times that on triangles)
  {
    const int j = lane >> 3;
    AccP a;
    accp_zero(a);
    if (valid >> j & 1) {
      const Elem& e = w.es[j];
      const int n = w.n[j], sh = w.sh[j];
      const double sx = w.sx[j], sy = w.sy[j];
      const double *xn = xr + RULE_OFF(n), *wn = wr + RULE_OFF(n);
      int left = (e.nn == 4) ? n : 3 * n, part = 0, i = 0, c = lane & 7;  // rows left, part, row, column
      if (c >= n) { c -= n; i++; left--; }
#pragma unroll 1
      while (left > 0) {
        double zeta = xn[i], eta = xn[c], wt = wn[i] * wn[c];
        if (e.nn != 4) {
          wt *= 1.0 + 0.25 * zeta + 0.25 * eta;
          lit_part_point(part, zeta, eta, zeta, eta);
        }
        smooth_near(e, L.k, w.rt, w.v0, w.v1, sx, sy, sh, zeta, eta, wt, a);
        c += 8;
        while (c >= n) { c -= n; i++; left--; }
        if (i >= n) { i -= n; part++; }
      }
    }
    accp_pack(a, &w.slot[lane * 19]);
  }
  __syncwarp();
#pragma unroll 1
  for (int i = lane; i < SMT_PAIRS * 19; i += 32) {
    const int j = i / 19, c = i - 19 * j;
    const double* v = &w.slot[8 * j * 19 + c];
    double s[2] = {0.0, 0.0};
#pragma unroll
    for (int q = 0; q < 8; q++) s[q & 1] += v[q * 19];
    w.tot[j][c] = s[0] + s[1];
  }
  __syncwarp();
  // smooth part
  int off[SMT_PAIRS + 1];
  off[0] = 0;
#pragma unroll
  for (int j = 0; j < SMT_PAIRS; j++)
    off[j + 1] = off[j] + ((valid >> j & 1) ? (w.es[j].nn == 4 ? P.nq4 : P.nq3) : 0);
  const int total = off[SMT_PAIRS];
  const int pj = (lane >> 2) & 3, pi = lane & 3, half = lane >> 4;
  int plo = 0, phi = 0;
#pragma unroll
  for (int j = 0; j < SMT_PAIRS; j++)
    if (pj == j) { plo = off[j]; phi = off[j + 1]; }
  cplx Gs = mk(0.0, 0.0), Hs = mk(0.0, 0.0);
#pragma unroll 1
  for (int base = 0; base < total; base += SMT_BUF) {
    const int end = min(total, base + SMT_BUF);
#pragma unroll 1
    for (int p = base + lane; p < end; p += 32) {
      int j = 0;
#pragma unroll
      for (int i = 1; i < SMT_PAIRS; i++)
        if (p >= off[i]) j = i;
      int o = 0;
#pragma unroll
      for (int i = 1; i < SMT_PAIRS; i++)
        if (j == i) o = off[i];
      cplx gw, hw;
      double z, n;
      smooth_point(w.es[j], L, P, M.tab, w.rt, w.sx[j], w.sy[j], p - o, w.rad + lane, 32, gw, hw, z, n);
      w.buf[p - base][0] = gw;
      w.buf[p - base][1] = hw;
    }
    __syncwarp();
    const int nn = w.es[pj].nn;
    const double* tq = (nn == 4) ? P.q4 : P.q3;
    for (int p = max(plo, base) + half; p < min(phi, end); p += 2) {
      double N[4];
      const double z = tq[3 * (p - plo)], n = tq[3 * (p - plo) + 1];
      if (nn == 4) bil_N4(z, n, N);
      else { lit_N3(z, n, N); N[3] = 0.0; }
      const double Ni = pi == 0 ? N[0] : pi == 1 ? N[1] : pi == 2 ? N[2] : N[3];
      Gs += w.buf[p - base][0] * Ni;
      Hs += w.buf[p - base][1] * Ni;
    }
    __syncwarp();
  }
  Gs.re += __shfl_down_sync(0xffffffffu, Gs.re, 16); Gs.im += __shfl_down_sync(0xffffffffu, Gs.im, 16);
  Hs.re += __shfl_down_sync(0xffffffffu, Hs.re, 16); Hs.im += __shfl_down_sync(0xffffffffu, Hs.im, 16);
  if (lane < 16) { w.sm[pj][pi][0] = Gs; w.sm[pj][pi][1] = Hs; }
  __syncwarp();
  // 8 lanes per pair store its G and H entries; the scalings are accp_finish's
  const int j = lane >> 3, it = lane & 7;
  if (j < np && (valid >> j & 1)) {
    const Elem& e = w.es[j];
    double gs = EL_I_FP, ss = 1.0, hs = EL_I_FP, st = 1.0, fs = EL_I_FP;
    if (e.nn != 4) {
      const double V[3] = {e.cw[0][0], e.cw[1][0], e.cw[2][0]};
      ss = 1.0 / 24.0 * vnorm3(V);
      st = 1.0 / 24.0;
      gs = ss * EL_I_FP;
      hs = st * EL_I_FP;
      fs = 0.0625 * EL_SQ3 * EL_I_SPSQ3;
    }
    const double* tot = w.tot[j];
    const double dFz = tot[17] * fs, dFe = tot[18] * fs;
    const unsigned pair = (unsigned)((long long)rr * A.ne + s0 + j);
    if (needs_gh(dFz, dFe)) {
      if (it == 0) {
        const unsigned slot = atomicAdd(gh_count, 1u);
        if (slot < gh_cap) gh_list[slot] = pair;
        else record_status(status, -900);
      }
    } else {
      const size_t N = (size_t)4 * A.ne, o = (size_t)row * N + (size_t)4 * (s0 + j);
      cplx v = (it < 4) ? mk(tot[2 * it], tot[2 * it + 1]) * gs + w.sm[j][it][0] * ss
                        : mk(tot[2 * it], tot[2 * it + 1]) * hs + w.sm[j][it - 4][1] * st;
      if (w.sh[j]) v = v * expi(L.vkx * w.sx[j] + L.vky * w.sy[j]);
      if (it < 4) ((cplx*)A.G)[o + it] = v;
      else ((cplx*)A.H)[o + it - 4] = v;
      if (it == 0) Fp[pair] = make_double3(tot[16] * fs, dFz, dFe);
    }
  }
}

__global__ void __launch_bounds__(SMT_WARPS * 32, SMT_BLOCKS)
    k_reg_smooth(AssembleArgs A, const __grid_constant__ QPLattice L, SmoothArgs M, int r0, int nr, double3* Fp,
                 unsigned* gh_list, unsigned* gh_count, unsigned gh_cap, unsigned* ip_list, unsigned* ip_count, int* status)
{
  if (!M.plan->on) return;
  extern __shared__ __align__(16) unsigned char smt_smem[];
  __shared__ double xr[RULE_TAB], wr[RULE_TAB];
  for (int i = threadIdx.x; i < RULE_TAB; i += SMT_WARPS * 32) { xr[i] = c_xr[i]; wr[i] = c_wr[i]; }
  __syncthreads();
  const int wib = threadIdx.x >> 5;
  const long long unit = (long long)blockIdx.x * SMT_WARPS + wib;
  if (unit >= (long long)((A.ne + SMT_PAIRS - 1) / SMT_PAIRS) * nr) return;  // uniform across the warp
  reg_smooth_unit(A, L, M, r0, unit, Fp, gh_list, gh_count, gh_cap, ip_list, ip_count, status,
                  reinterpret_cast<SmoothWarp*>(smt_smem)[wib], xr, wr, threadIdx.x & 31);
}

// Near-singular pair w of the chunk starting at pair p0, by the whole CTA: the 64 x 64 rule for the
// nearest image and the solid angle, the smooth points by the first threads.
__device__ __forceinline__ void gh_smooth_pair(const AssembleArgs& A, const QPLattice& L, const SmoothPlan& P,
                                               const cplx* __restrict__ tab, long long p0, long long w, double3* Fp,
                                               double (*red)[19], const double* xh, const double* wh)
{
  const PairIdx q = pair_of(p0 + w, A.ne);
  int tnn;
  double rt[3], vtz[3], vte[3];
  target_info(A.geo, A.sid, q.t, q.tn, rt, vtz, vte, tnn);
  Elem es;
  load_elem(A.geo, abs(A.sid[q.s]), es);
  const double v[3] = {es.cr[0][0] - rt[0], es.cr[1][0] - rt[1], es.cr[2][0] - rt[2]};
  double sx, sy;
  const int sh = smooth_shift(L, v, &sx, &sy);
  AccP a;
  accp_zero(a);
  const int npts = (es.nn == 4) ? 4096 : 3 * 4096;
#pragma unroll 1
  for (int k = threadIdx.x; k < npts; k += blockDim.x) {
    double z, e, wt;
    rule_point(es.nn, 64, xh, wh, k, z, e, wt);
    smooth_near(es, L.k, rt, vtz, vte, sx, sy, sh, z, e, wt, a);
  }
  for (int i = 0; i < 4; i++) { a.G[i] = a.G[i] * EL_I_FP; a.H[i] = a.H[i] * EL_I_FP; }
  const int nq = (es.nn == 4) ? P.nq4 : P.nq3;
  double rad[SMT_LMAX + 2];
#pragma unroll 1
  for (int k = threadIdx.x; k < nq; k += blockDim.x) {
    cplx gw, hw;
    double z, e, N[4];
    smooth_point(es, L, P, tab, rt, sx, sy, k, rad, 1, gw, hw, z, e);
    if (es.nn == 4) bil_N4(z, e, N);
    else { lit_N3(z, e, N); N[3] = 0.0; }
    for (int i = 0; i < 4; i++) { a.G[i] += gw * N[i]; a.H[i] += hw * N[i]; }
  }
  double s[19];
  accp_pack(a, s);
  warp_sum_arr<19>(s);
  const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (lane == 0)
    for (int i = 0; i < 19; i++) red[wid][i] = s[i];
  __syncthreads();
  if (wid == 0) {
    for (int i = 0; i < 19; i++) s[i] = (lane < (int)(blockDim.x >> 5)) ? red[lane][i] : 0.0;
    warp_sum_arr<19>(s);
    accp_unpack(s, a);
    if (sh) {
      const cplx ph = expi(L.vkx * sx + L.vky * sy);
      for (int i = 0; i < 4; i++) { a.G[i] = a.G[i] * ph; a.H[i] = a.H[i] * ph; }
    }
    cplx CC[9], dCz[9], dCe[9];
    accp_finish(es, a, CC, dCz, dCe);
    store_pair(A, q.row, q.s, CC, dCz, dCe, Fp, w, lane);
  }
  __syncthreads();
}

__global__ void __launch_bounds__(256, 2) k_gh_smooth(AssembleArgs A, const __grid_constant__ QPLattice L, SmoothArgs M,
                                                      long long p0, double3* Fp, const unsigned* gh_list,
                                                      const unsigned* gh_count, unsigned gh_cap)
{
  const SmoothPlan& P = *M.plan;
  if (!P.on) return;
  __shared__ double red[8][19];
  __shared__ double xh[64], wh[64];
  if (threadIdx.x < 64) { xh[threadIdx.x] = c_xh[threadIdx.x]; wh[threadIdx.x] = c_wh[threadIdx.x]; }
  __syncthreads();
  const unsigned n = min(*gh_count, gh_cap);
  for (unsigned it = blockIdx.x; it < n; it += gridDim.x) gh_smooth_pair(A, L, P, M.tab, p0, gh_list[it], Fp, red, xh, wh);
}

// Self pair of row `row`, by the whole CTA: the polar rule for the nearest image and the solid angles,
// the smooth points by the first threads.  The normal derivative of the nearest image uses
// K . W = r cos(theta) sin(theta) b.(d x C) (bdc) of the bilinear map, as the interior self rule does
// (zero on planes).
__device__ __forceinline__ void self_smooth_row(const AssembleArgs& A, const QPLattice& L, const SmoothPlan& P,
                                                const cplx* __restrict__ tab, int row, double3* Fself, double (*red)[24],
                                                const double* xl, const double* wl, const double* xh, const double* wh)
{
  const int t = row >> 2, tn = row & 3;
  const int at = abs(A.sid[t]);
  SelfInfo S;
  self_setup(A.geo, at, tn, mk(L.k, 0.0), S);
  if (tn == 3 && S.e.nn == 3) return;
  const Elem& e = S.e;
  double v[24];
  for (int i = 0; i < 24; i++) v[i] = 0.0;
  const double bdc = e.cr[0][1] * e.cw[0][2] + e.cr[1][1] * e.cw[1][2] + e.cr[2][1] * e.cw[2][2];
  // one azimuth of the polar rule at a time: 12 radial points share its trigonometry
  const int nth = S.P.nsub * 128;
#pragma unroll 1
  for (int q = threadIdx.x; q < nth * 4; q += blockDim.x) {
    const int tq = q >> 2, ir0 = (q & 3) * 3;
    const int j = tq >> 7, m2 = tq & 127;
    double theta, wt;
    polar_theta(S.P, j, m2, xh, wh, theta, wt);
    const double rm = polar_rm(S.P, j, theta);
    double sth, cth;
    sincos(theta, &sth, &cth);
#pragma unroll 1
    for (int ir = ir0; ir < ir0 + 3; ir++) {
      const double r = 0.5 * rm * (xl[ir] + 1.0);
      const double w = wt * 0.5 * rm * wl[ir];
      const double zeta = r * cth + S.zt, eta = r * sth + S.et;
      double K[3], N[4];
      self_K(S, r, cth, sth, K);
      self_N(S, zeta, eta, N);
      const double K2 = dot3(K, K), iK = rsqrt_(K2);
      const double kr = L.k * r * K2 * iK;
      const cplx ce = expi(kr);
      const cplx g = ce * (w * EL_I_FP * iK * self_aW(S, zeta, eta));
      for (int i = 0; i < 4; i++) acc_put(v, i, g * N[i]);
      if (S.curved) {
        const cplx h = (ce * mk(-1.0, kr)) * (w * EL_I_FP * bdc * cth * sth * iK * iK * iK);
        for (int i = 0; i < 4; i++) acc_put(v, 4 + i, h * N[i]);
      }
    }
  }
  if (S.bil && S.curved) {
    const double h = EL_CDFH;
    const double cz[5] = {S.zt, S.zt + h, S.zt - h, S.zt, S.zt};
    const double ce[5] = {S.et, S.et, S.et, S.et + h, S.et - h};
#pragma unroll 1
    for (int c = 0; c < 5; c++) {
      const double f = bil_self_F(e, cz[c], ce[c], xl, wl, xh, wh, threadIdx.x, blockDim.x);
      if (c == 0) v[16] += f;
      else if (c == 1) v[17] += f;
      else if (c == 2) v[18] += f;
      else if (c == 3) v[19] += f;
      else v[20] += f;
    }
  }
  const double* rt = A.geo + (size_t)at * GEO_STRIDE + GEO_REN + tn * 3;
  const int nq = S.bil ? P.nq4 : P.nq3;
  // the smooth rules' weights sum to 4 (quads) and 12 (triangles); the polar rule covers 4 and
  // 3 sqrt(3) / 4
  const double sc = S.bil ? 1.0 : EL_SQ3 / 16.0;
  double rad[SMT_LMAX + 2];
#pragma unroll 1
  for (int k = threadIdx.x; k < nq; k += blockDim.x) {
    cplx gw, hw;
    double z, n, N[4];
    smooth_point(e, L, P, tab, rt, 0.0, 0.0, k, rad, 1, gw, hw, z, n);
    self_N(S, z, n, N);
    for (int i = 0; i < 4; i++) { acc_put(v, i, gw * (sc * N[i])); acc_put(v, 4 + i, hw * (sc * N[i])); }
  }
  warp_sum_arr<24>(v);
  const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (lane == 0)
    for (int i = 0; i < 24; i++) red[wid][i] = v[i];
  __syncthreads();
  if (wid != 0) return;
  for (int i = 0; i < 24; i++) v[i] = (lane < SELF_THREADS / 32) ? red[lane][i] : 0.0;
  warp_sum_arr<24>(v);
  if (lane != 0) return;
  cplx CC[9], dCz[9], dCe[9];
  self_per_combine(S, v, CC, dCz, dCe);
  store_pair(A, row, t, CC, dCz, dCe, Fself, row, -1);
}

__global__ void __launch_bounds__(SELF_THREADS, 2) k_self_smooth(AssembleArgs A, const __grid_constant__ QPLattice L,
                                                                 SmoothArgs M, double3* Fself)
{
  const SmoothPlan& P = *M.plan;
  if (!P.on) return;
  __shared__ double red[SELF_THREADS / 32][24];
  __shared__ double xl[12], wl[12], xh[64], wh[64];
  if (threadIdx.x < 12) { xl[threadIdx.x] = c_xl[threadIdx.x]; wl[threadIdx.x] = c_wl[threadIdx.x]; }
  if (threadIdx.x < 64) { xh[threadIdx.x] = c_xh[threadIdx.x]; wh[threadIdx.x] = c_wh[threadIdx.x]; }
  __syncthreads();
  self_smooth_row(A, L, P, M.tab, blockIdx.x, Fself, red, xl, wl, xh, wh);
}
