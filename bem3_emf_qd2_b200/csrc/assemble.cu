// assemble.cu -- sm_100a kernels for the coefficient-matrix assembly of one domain
// (the reference's create_cmatrix_domain, d3qd2_src/d3qd2_solve_bieq.c:165-256).
//
// Output layout is the reference's (d3qd2_solve_bieq.c:213-236), N = 4 * Ne_d:
//   G, H   [N][N]     row (t,tn) = 4 t + tn, column (s,i) = 4 s + i        (complex)
//   dG, dH [2N][N]    row 2 (4 t + tn) + {0: d/dt_zeta, 1: d/dt_eta}       (complex)
//   dF     [N][3]     (F or 1+F, dF/dt_zeta, dF/dt_eta)                   (double)
// with 0-based t, s indexing sb[did].sid.  Rows tn = 3 of triangles are left zero, as in
// the reference.
//
// Work decomposition (all FP64, no tensor cores -- none of this is a contraction):
//   k_*_smooth     : the periodic domain's pairs by the nearest image and a table of the rest
//                    (assemble_smooth.cuh); what it leaves, and domains without a table:
//   k_self_periodic / k_self_interior : one CTA per self pair (t == s), polar rule;
//   k_reg_periodic : one warp per 2 regular pairs, lanes over the 144 (quad) / 432 (triangle)
//                    Gauss points, one quasi-periodic Green's function per point;
//   k_reg_interior : one thread per regular pair (free-space kernel), a warp per 32 sources of a row;
//   k_gh_*         : pairs whose GL dF/dv exceeds CBD_SDF, recomputed with the 64x64 rule from a
//                    compacted device work list (no host round trip);
//   k_rowsum       : deterministic per-row sums of F, dF/dt over s, H diagonal += (1+)F.
// Regular pairs run in row chunks so that the per-pair F scratch stays bounded.
#include <cuda_runtime.h>
#include <stdint.h>
#include <stdio.h>
#include <string.h>

#include <vector>

#include "self.cuh"
#include "smooth.cuh"
#include "bem3_internal.h"

// ------------------------------------------------------------------------------------------
// Constant tables: Gauss-Legendre nodes (12, 64) and the open-domain lattice.
__constant__ double c_xl[12], c_wl[12], c_xh[64], c_wh[64];
__constant__ double c_xr[RULE_TAB], c_wr[RULE_TAB];  // the rules of 6 to 12 points
__constant__ double c_xs[SELF_NLOG], c_ws[SELF_NLOG];

// ------------------------------------------------------------------------------------------
__device__ __forceinline__ double warp_sum(double v)
{
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ int warp_min_i(int v)
{
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = min(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
template <int N>
__device__ __forceinline__ void warp_sum_arr(double* v)
{
#pragma unroll
  for (int i = 0; i < N; i++) v[i] = warp_sum(v[i]);
}

__device__ __forceinline__ void record_status(int* status, int err)
{
  if (err < 0) atomicCAS(status, 0, err);
}

struct PairIdx {
  int row, s, t, tn;
};
__device__ __forceinline__ PairIdx pair_of(long long p, int ne)
{
  PairIdx q;
  q.row = (int)(p / ne);
  q.s = (int)(p - (long long)q.row * ne);
  q.t = q.row >> 2;
  q.tn = q.row & 3;
  return q;
}

__device__ __forceinline__ void target_info(const double* __restrict__ geo, const int* __restrict__ sid, int t, int tn,
                                            double* rt, double* vtz, double* vte, int& tnn)
{
  int at = abs(sid[t]);
  Elem et;
  load_elem(geo, at, et);
  tnn = et.nn;
  node_tangents(et, tn, vtz, vte);
  const double* g = geo + (size_t)at * GEO_STRIDE + GEO_REN + tn * 3;
  rt[0] = g[0]; rt[1] = g[1]; rt[2] = g[2];
}

// AccP <-> flat array (19 doubles)
__device__ __forceinline__ void accp_pack(const AccP& a, double* v)
{
  for (int i = 0; i < 4; i++) { v[2 * i] = a.G[i].re; v[2 * i + 1] = a.G[i].im; v[8 + 2 * i] = a.H[i].re; v[9 + 2 * i] = a.H[i].im; }
  v[16] = a.F; v[17] = a.dF0; v[18] = a.dF1;
}
__device__ __forceinline__ void accp_unpack(const double* v, AccP& a)
{
  for (int i = 0; i < 4; i++) { a.G[i] = mk(v[2 * i], v[2 * i + 1]); a.H[i] = mk(v[8 + 2 * i], v[9 + 2 * i]); }
  a.F = v[16]; a.dF0 = v[17]; a.dF1 = v[18];
}
// A complex matrix whose entries may be stored 16 bytes at a time: a caller's array of doubles need not
// start on such a boundary.
__host__ __device__ __forceinline__ bool wide_cplx(const double* m) { return (reinterpret_cast<uintptr_t>(m) & 15) == 0; }
static inline bool wide_outputs(const AssembleArgs& A)
{
  return wide_cplx(A.G) && wide_cplx(A.H) && wide_cplx(A.dG) && wide_cplx(A.dH);
}
// Store one pair's coefficients in the reference layout.  Done by lanes of a warp (lane l
// stores item l) or by a single thread (lane = -1 stores all).
__device__ __forceinline__ void store_pair(const AssembleArgs& A, int row, int s, const cplx* CC, const cplx* dCz,
                                           const cplx* dCe, double3* Fp, long long fidx, int lane)
{
  const size_t N = (size_t)4 * A.ne;
  const size_t col = (size_t)4 * s;
  cplx* G = (cplx*)A.G;
  cplx* H = (cplx*)A.H;
  cplx* dG = (cplx*)A.dG;
  cplx* dH = (cplx*)A.dH;
  for (int it = (lane < 0 ? 0 : lane); it < 25; it += (lane < 0 ? 1 : 32)) {
    if (it < 4) G[(size_t)row * N + col + it] = CC[it];
    else if (it < 8) H[(size_t)row * N + col + it - 4] = CC[it];
    else if (it < 12) { if (dG) dG[(size_t)(2 * row) * N + col + it - 8] = dCz[it - 8]; }
    else if (it < 16) { if (dG) dG[(size_t)(2 * row + 1) * N + col + it - 12] = dCe[it - 12]; }
    else if (it < 20) { if (dH) dH[(size_t)(2 * row) * N + col + it - 16] = dCz[it - 12]; }
    else if (it < 24) { if (dH) dH[(size_t)(2 * row + 1) * N + col + it - 20] = dCe[it - 16]; }
    else Fp[fidx] = make_double3(CC[8].re, dCz[8].re, dCe[8].re);
  }
}

// ==========================================================================================
#ifndef REGP_MIN_BLOCKS
#define REGP_MIN_BLOCKS 2  // 2 x 256 threads per SM: 128 registers (measured fastest with register-resident sums)
#endif
// Per-warp pair data in shared memory: the source element and the collocation node with its
// tangents, read by all lanes.  With them and the lanes' sums in shared memory, only a lane's
// current quadrature point stays live in registers across the (out-of-line) lattice sums.
struct RegWarp {
  Elem es;
  double rt[3], vtz[3], vte[3];
};
#define REGP_PAIRS 2  // pairs per warp: 2 x 144 Gauss points = 9 per lane, no ragged last step
#define REGP_SMEM_BYTES (sizeof(RegWarp) * 8 * REGP_PAIRS + sizeof(AccP) * 256 * REGP_PAIRS)

// One warp's unit of regular periodic work: the pairs first, first + 1, ... (REGP_PAIRS of them,
// those < np) of the chunk that starts at pair p0 of the domain, or of the list of pairs of that
// chunk (list != nullptr, np entries).  Lane l takes the points l, l + 32,
// ... of the pairs' concatenated point lists.  sw: the warp's REGP_PAIRS pair slots; sacc: the
// block's per-thread accumulators (shared memory).
__device__ __forceinline__ void reg_periodic_unit(const AssembleArgs& A, const QPLattice& L, long long p0, long long np,
                                                  long long first, const unsigned* list, double3* Fp, unsigned* gh_list,
                                                  unsigned* gh_count, unsigned gh_cap, int* status, RegWarp* sw,
                                                  AccP (*sacc)[256], int lane)
{
  int npts[REGP_PAIRS];
  long long pidx[REGP_PAIRS];  // pair within the chunk
  PairIdx q[REGP_PAIRS];
  __syncwarp();  // a warp that runs several units reuses its slots: the last unit's reads are done
#pragma unroll
  for (int j = 0; j < REGP_PAIRS; j++) {
    npts[j] = 0;
    pidx[j] = first + j;
    if (first + j >= np) continue;
    if (list) pidx[j] = list[first + j];
    q[j] = pair_of(p0 + pidx[j], A.ne);
    const int at = abs(A.sid[q[j].t]);
    const int tnn = (int)A.geo[(size_t)at * GEO_STRIDE + GEO_NN];
    if ((q[j].tn == 3 && tnn == 3) || q[j].s == q[j].t) continue;
    RegWarp& W = sw[j];
    if (lane == 0) {
      int tn_unused;
      target_info(A.geo, A.sid, q[j].t, q[j].tn, W.rt, W.vtz, W.vte, tn_unused);
      load_elem(A.geo, abs(A.sid[q[j].s]), W.es);
    }
    const int sn = (int)A.geo[(size_t)abs(A.sid[q[j].s]) * GEO_STRIDE + GEO_NN];
    npts[j] = (sn == 4) ? 144 : 432;
    accp_zero(sacc[j][threadIdx.x]);
  }
  __syncwarp();
  // a list's order varies from run to run: each of its pairs starts at lane 0, whatever its neighbour,
  // so that its sums are the same
  const int off1 = list ? (npts[0] + 31) & ~31 : npts[0];
  const int ntot = off1 + npts[1];
  int err = 0, nterms = 0;
  for (int k = lane; k < ntot; k += 32) {
    const int j = (k < off1) ? 0 : 1;
    const int kk = j ? k - off1 : k;
    if (kk >= npts[j]) continue;
    const RegWarp& W = sw[j];
    double z, e, wt;
    rule_point(W.es.nn, 12, c_xl, c_wl, kk, z, e, wt);
    int e2 = accp_point(W.es, L, W.rt, W.vtz, W.vte, z, e, wt, sacc[j][threadIdx.x]);
    if (e2 < 0) err = e2;
    else nterms += e2;
  }
  err = warp_min_i(err);
  if (lane == 0) record_status(status, err);
  if (A.terms) {
    double tc = warp_sum((double)nterms);
    if (lane == 0) atomicAdd(A.terms, (unsigned long long)tc);
  }
#pragma unroll 1
  for (int j = 0; j < REGP_PAIRS; j++) {
    if (npts[j] == 0) continue;  // uniform across the warp
    // Warp totals of the 19 sums (AccP is 19 doubles: G, H interleaved re/im, F, dF0, dF1): lane
    // i < 19 adds component i over the warp's 32 shared-memory slots, then writes it to slot 0,
    // which every lane reads for the one item it stores.  No per-thread arrays: the scaled
    // coefficients never leave registers or shared memory.
    double* acc = reinterpret_cast<double*>(&sacc[j][threadIdx.x & ~31]);
    static_assert(sizeof(AccP) == 19 * sizeof(double), "AccP is read as 19 doubles");
    __syncwarp();  // every lane's last accumulation is visible to the others
    double tot = 0.0;
    if (lane < 19) {
      double s0 = 0.0, s1 = 0.0, s2 = 0.0, s3 = 0.0;
#pragma unroll
      for (int t = 0; t < 32; t += 4) {
        s0 += acc[(t + 0) * 19 + lane];
        s1 += acc[(t + 1) * 19 + lane];
        s2 += acc[(t + 2) * 19 + lane];
        s3 += acc[(t + 3) * 19 + lane];
      }
      tot = (s0 + s1) + (s2 + s3);
    }
    __syncwarp();
    if (lane < 19) acc[lane] = tot;
    __syncwarp();
    // the scalings of accp_finish: quads as summed; triangles G |W| / 24, H / 24
    double gs = 1.0, hs = 1.0, fs = EL_I_FP;
    if (sw[j].es.nn != 4) {
      const double V[3] = {sw[j].es.cw[0][0], sw[j].es.cw[1][0], sw[j].es.cw[2][0]};
      gs = 1.0 / (24.0) * vnorm3(V);
      hs = 1.0 / (24.0);
      fs = 0.0625 * EL_SQ3 * EL_I_SPSQ3;
    }
    const double dFz = acc[17] * fs, dFe = acc[18] * fs;
    const long long pi = j ? pidx[REGP_PAIRS - 1] : pidx[0];
    if (needs_gh(dFz, dFe)) {
      if (lane == 0) {
        unsigned slot = atomicAdd(gh_count, 1u);
        if (slot < gh_cap) gh_list[slot] = (unsigned)pi;
        else record_status(status, -900);
      }
      continue;
    }
    // lane it stores item it of store_pair's order: G[0..3], H[0..3], the (zero) dG and dH rows, F
    const size_t N = (size_t)4 * A.ne, col = (size_t)4 * q[j].s, row = (size_t)q[j].row;
    const int it = lane;
    if (it < 4) {
      ((cplx*)A.G)[row * N + col + it] = mk(acc[2 * it] * gs, acc[2 * it + 1] * gs);
    } else if (it < 8) {
      ((cplx*)A.H)[row * N + col + it - 4] = mk(acc[2 * it] * hs, acc[2 * it + 1] * hs);
    } else if (it < 16) {
      if (A.dG) ((cplx*)A.dG)[(2 * row + (it >= 12)) * N + col + (it & 3)] = mk(0, 0);
    } else if (it < 24) {
      if (A.dH) ((cplx*)A.dH)[(2 * row + (it >= 20)) * N + col + (it & 3)] = mk(0, 0);
    } else if (it == 24) {
      Fp[pi] = make_double3(acc[16] * fs, dFz, dFe);
    }
    __syncwarp();  // slot 0 is rewritten by the next pair's accumulation only after every read
  }
}

// Regular periodic pairs of one chunk summed point by point: one warp per REGP_PAIRS pairs, striding
// over all pairs of the chunk, or (plan on) over the list of pairs that the tabulated kernel left.
__global__ void __launch_bounds__(256, REGP_MIN_BLOCKS) k_reg_periodic(AssembleArgs A, const __grid_constant__ QPLattice L,
                                                                       const SmoothPlan* plan, const unsigned* list,
                                                                       const unsigned* nlist, long long p0, long long np,
                                                                       double3* Fp, unsigned* gh_list, unsigned* gh_count,
                                                                       unsigned gh_cap, int* status)
{
  extern __shared__ __align__(16) unsigned char regp_smem[];  // REGP_SMEM_BYTES
  RegWarp(*sw)[REGP_PAIRS] = reinterpret_cast<RegWarp(*)[REGP_PAIRS]>(regp_smem);
  AccP(*sacc)[256] = reinterpret_cast<AccP(*)[256]>(regp_smem + sizeof(RegWarp) * 8 * REGP_PAIRS);
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  const bool on = plan && plan->on;
  if (on) np = *nlist;
  const long long stride = (long long)gridDim.x * (blockDim.x >> 5) * REGP_PAIRS;
  for (long long first = (((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5) * REGP_PAIRS; first < np; first += stride)
    reg_periodic_unit(A, L, p0, np, first, on ? list : nullptr, Fp, gh_list, gh_count, gh_cap, status, sw[wib], sacc, lane);
}

// Near-singular periodic pair w of the chunk starting at pair p0, 64x64 rule, by the whole CTA
// (256 threads; red, serr: its shared reduction slots).  Every thread of the CTA calls it.
__device__ __forceinline__ void gh_periodic_pair(const AssembleArgs& A, const QPLattice& L, long long p0, long long w,
                                                 double3* Fp, int* status, double (*red)[19], int* serr)
{
  {
    PairIdx q = pair_of(p0 + w, A.ne);
    int tnn;
    double rt[3], vtz[3], vte[3];
    target_info(A.geo, A.sid, q.t, q.tn, rt, vtz, vte, tnn);
    Elem es;
    load_elem(A.geo, abs(A.sid[q.s]), es);
    AccP a;
    accp_zero(a);
    int err = 0;
    const int npts = (es.nn == 4) ? 4096 : 3 * 4096;
    for (int k = threadIdx.x; k < npts; k += blockDim.x) {
      double z, e, wt;
      rule_point(es.nn, 64, c_xh, c_wh, k, z, e, wt);
      int e2 = accp_point(es, L, rt, vtz, vte, z, e, wt, a);
      if (e2 < 0) err = e2;
    }
    double v[19];
    accp_pack(a, v);
    warp_sum_arr<19>(v);
    err = warp_min_i(err);
    int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (lane == 0) { for (int i = 0; i < 19; i++) red[wid][i] = v[i]; serr[wid] = err; }
    __syncthreads();
    if (wid == 0) {
      for (int i = 0; i < 19; i++) v[i] = (lane < 8) ? red[lane][i] : 0.0;
      warp_sum_arr<19>(v);
      int e3 = warp_min_i(lane < 8 ? serr[lane] : 0);
      if (lane == 0) record_status(status, e3);
      accp_unpack(v, a);
      cplx CC[9], dCz[9], dCe[9];
      accp_finish(es, a, CC, dCz, dCe);
      store_pair(A, q.row, q.s, CC, dCz, dCe, Fp, w, lane);
    }
    __syncthreads();
  }
}

// Near-singular periodic pairs of one chunk: one CTA per listed pair.  The list holds at most
// gh_cap entries (the counter keeps counting past it; the regular kernel then reports -900).
__global__ void __launch_bounds__(256, 2) k_gh_periodic(AssembleArgs A, const __grid_constant__ QPLattice L, long long p0, double3* Fp,
                                                     const unsigned* gh_list, const unsigned* gh_count, unsigned gh_cap,
                                                     int* status)
{
  __shared__ double red[8][19];
  __shared__ int serr[8];
  const unsigned n = min(*gh_count, gh_cap);
  for (unsigned it = blockIdx.x; it < n; it += gridDim.x) gh_periodic_pair(A, L, p0, gh_list[it], Fp, status, red, serr);
}

// ==========================================================================================
// Regular interior pairs: one thread per pair, a warp's 32 pairs being consecutive sources of one row.
//
// The n x n rule (three of them on triangles; n = 6 to 12, rule_order) is walked by rows of the first coordinate a.  Along a
// row the position, the normal, their products with the node's tangents and the shape functions are
// linear in the second coordinate b:
//   r - rt = P + Q b,  W = C + D b,  N_i = al_i + be_i b,
// so a point adds a few scalars to moments sum f b^m instead of evaluating six integrands and four
// shape functions each; the moments become shape-function sums once per row, kept in shared memory
// (48 doubles a thread: in registers they would leave room for 8 warps an SM).  With q = (ikR - 1) e^{ikR}
// / R^3 and e5 = ((kR)^2 + 3 (ikR - 1)) e^{ikR} (R.W) / R^5 the integrands are
//   G = e |W| / R,  H = q (R.W),  dG_v = q |W| (R.v),  dH_v = e5 (R.v) - q (W.v).
// e^{ikR} along a row is e^{ikR0} (its middle) times a Taylor sum in k (R - R0), without reductions and
// branches, where every element of the warp is smaller than the sums' range.  At the end the warp writes
// its row segments of each matrix from shared memory, 512 contiguous bytes an instruction.
#define REGI_WARPS 1  // a CTA's warps would wait for the one whose pairs take the most points
#define REGI_LD 33  // leading dimension of the sums (pad: the transposed read of the stores)
#define REGI_SMEM (48 * REGI_LD + 21 * 32 + 10)  // doubles a warp: the sums, the lanes' elements, rt, v0, v1
#define REGI_SMEM_BYTES (sizeof(double) * REGI_SMEM * REGI_WARPS)
// Ranges of the Taylor sums: cos and sin to x^18 and x^17 (next terms below 1e-17 for |x| <= 0.9), e^-y
// to y^10 (below 1e-17 for |y| <= 0.12).
#define REGI_XMAX 0.9
#define REGI_YMAX 0.12

__device__ __forceinline__ cplx taylor_cis(double x)
{
  const double t = x * x;
  double c = -1.0 / 6402373705728000.0, s = 1.0 / 355687428096000.0;
  c = fma(c, t, 1.0 / 20922789888000.0);
  s = fma(s, t, -1.0 / 1307674368000.0);
  c = fma(c, t, -1.0 / 87178291200.0);
  s = fma(s, t, 1.0 / 6227020800.0);
  c = fma(c, t, 1.0 / 479001600.0);
  s = fma(s, t, -1.0 / 39916800.0);
  c = fma(c, t, -1.0 / 3628800.0);
  s = fma(s, t, 1.0 / 362880.0);
  c = fma(c, t, 1.0 / 40320.0);
  s = fma(s, t, -1.0 / 5040.0);
  c = fma(c, t, -1.0 / 720.0);
  s = fma(s, t, 1.0 / 120.0);
  c = fma(c, t, 1.0 / 24.0);
  s = fma(s, t, -1.0 / 6.0);
  c = fma(c, t, -0.5);
  return mk(fma(c, t, 1.0), fma(s, t * x, x));
}
__device__ __forceinline__ double taylor_expm(double y)  // e^{-y}
{
  double s = 1.0 / 3628800.0;
  s = fma(s, y, -1.0 / 362880.0);
  s = fma(s, y, 1.0 / 40320.0);
  s = fma(s, y, -1.0 / 5040.0);
  s = fma(s, y, 1.0 / 720.0);
  s = fma(s, y, -1.0 / 120.0);
  s = fma(s, y, 1.0 / 24.0);
  s = fma(s, y, -1.0 / 6.0);
  s = fma(s, y, 0.5);
  s = fma(s, y, -1.0);
  return fma(s, y, 1.0);
}

// Moments of one row: with b the second coordinate and w its weight
struct RegiRow {
  cplx g0, g1;          // G:        sum g, g b
  cplx h0, h1;          // H
  cplx a0, a1, a2;      // q |W|:    sum, b, b^2
  cplx e0, e1, e2;      // e5
  cplx q0, q1, q2;      // q
  double F, s0, s1, t0, t1;  // (R.W) / R^3; 3 (R.W) / R^5 and 1 / R^3: sum, b
};

// Row a (coordinate a of part `part` of a triangle's rule) of element e seen from rt: the linear forms
// and the weight factor.
struct RegiLine {
  double P[3], Q[3], C[3], D[3], wf0, wf1;
};
// Its shape functions N_i = al[i] + be[i] b.
__device__ __forceinline__ void regi_shape(bool tri, int part, double a, double* al, double* be)
{
  if (!tri) {
    const double i_a = 1.0 / EL_P44_N;
#pragma unroll
    for (int i = 0; i < 4; i++) {
      al[i] = (i == 0 || i == 3) ? 0.25 * (1.0 - a * i_a) : 0.25 * (1.0 + a * i_a);
      be[i] = (i < 2) ? -al[i] * i_a : al[i] * i_a;
    }
    return;
  }
  double z0, z1, n0, n1;
  regi_part(part, a, z0, z1, n0, n1);
  const double h = 0.5 / EL_P34_N0 / 3.0;
  al[0] = 1.0 / 3.0 - h * (z0 + EL_SQ3 * n0); be[0] = -h * (z1 + EL_SQ3 * n1);
  al[1] = 1.0 / 3.0 + 2.0 * h * z0;           be[1] = 2.0 * h * z1;
  al[2] = 1.0 / 3.0 - h * (z0 - EL_SQ3 * n0); be[2] = -h * (z1 - EL_SQ3 * n1);
  al[3] = be[3] = 0.0;
}
__device__ __forceinline__ void regi_line(const Elem& e, const double* rt, int part, double a, RegiLine& y)
{
  if (e.nn == 4) {
    y.wf0 = 1.0;
    y.wf1 = 0.0;
#pragma unroll
    for (int i = 0; i < 3; i++) {
      y.P[i] = e.cr[i][0] + e.cr[i][1] * a - rt[i];
      y.Q[i] = e.cr[i][2] + e.cr[i][3] * a;
      y.C[i] = e.cw[i][0] + e.cw[i][1] * a;
      y.D[i] = e.cw[i][2];
    }
    return;
  }
  double z0, z1, n0, n1;
  regi_part(part, a, z0, z1, n0, n1);
  y.wf0 = 1.0 + 0.25 * a;
  y.wf1 = 0.25;
#pragma unroll
  for (int i = 0; i < 3; i++) {
    y.P[i] = e.cr[i][0] + e.cr[i][1] * z0 + e.cr[i][2] * n0 - rt[i];
    y.Q[i] = e.cr[i][1] * z1 + e.cr[i][2] * n1;
    y.C[i] = e.cw[i][0];
    y.D[i] = 0.0;
  }
}

// Points j0 .. j1 - 1 of a row (nodes xs, weights ws).  SHORT: the Taylor sums' range holds.
template <bool SHORT>
__device__ __forceinline__ void regi_row(const RegiLine& line, const double* xs, const double* ws, int j0, int j1, bool tri,
                                         double kre, double kim, RegiRow& m)
{
  const double *P = line.P, *Q = line.Q, *C = line.C, *D = line.D;
  cplx e0 = mk(1.0, 0.0);
  double R0 = 0.0;
  if (SHORT) {
    R0 = vnorm3(P);
    e0 = expi(kre * R0) * exp(-kim * R0);
  }
  const bool damped = kim != 0.0;
#pragma unroll 1
  for (int j = j0; j < j1; j++) {
    const double b = xs[j], w = ws[j] * fma(line.wf1, b, line.wf0);
    const double x = fma(Q[0], b, P[0]), y = fma(Q[1], b, P[1]), z = fma(Q[2], b, P[2]);
    const double Wx = fma(D[0], b, C[0]), Wy = fma(D[1], b, C[1]), Wz = fma(D[2], b, C[2]);
    const double R2 = x * x + y * y + z * z;
    const double iR = rsqrt_(R2), R = R2 * iR, i2 = iR * iR;
    const double RW = x * Wx + y * Wy + z * Wz;
    double wG = w;
    if (!tri) {
      const double W2 = Wx * Wx + Wy * Wy + Wz * Wz;
      wG = w * (W2 * rsqrt_(W2));
    }
    const cplx kR = mk(kre * R, kim * R);
    cplx u;
    if (SHORT) {
      const double d = R - R0;
      u = e0 * taylor_cis(kre * d);
      if (damped) u = u * taylor_expm(kim * d);
    } else {
      u = expi(kR.re);
      if (damped) u = u * exp(-kR.im);
    }
    const double w3 = i2 * iR;
    const cplx g = u * (wG * iR);
    const cplx cb = mk(-kR.im - 1.0, kR.re);
    const cplx q = (cb * u) * w3;
    const cplx qa = q * wG, qw = q * w;
    const cplx h = qw * RW;
    const cplx k3 = mk(kR.re * kR.re - kR.im * kR.im + 3.0 * cb.re, 2.0 * kR.re * kR.im + 3.0 * cb.im);
    const double t5 = w3 * w, s5 = t5 * i2 * RW;
    const cplx e5 = (k3 * u) * s5;
    const double b2 = b * b;
    m.g0 += g; m.g1.re = fma(g.re, b, m.g1.re); m.g1.im = fma(g.im, b, m.g1.im);
    m.h0 += h; m.h1.re = fma(h.re, b, m.h1.re); m.h1.im = fma(h.im, b, m.h1.im);
    m.a0 += qa; m.a1.re = fma(qa.re, b, m.a1.re); m.a1.im = fma(qa.im, b, m.a1.im);
    m.a2.re = fma(qa.re, b2, m.a2.re); m.a2.im = fma(qa.im, b2, m.a2.im);
    m.e0 += e5; m.e1.re = fma(e5.re, b, m.e1.re); m.e1.im = fma(e5.im, b, m.e1.im);
    m.e2.re = fma(e5.re, b2, m.e2.re); m.e2.im = fma(e5.im, b2, m.e2.im);
    m.q0 += qw; m.q1.re = fma(qw.re, b, m.q1.re); m.q1.im = fma(qw.im, b, m.q1.im);
    m.q2.re = fma(qw.re, b2, m.q2.re); m.q2.im = fma(qw.im, b2, m.q2.im);
    m.F = fma(t5, RW, m.F);
    const double s3 = 3.0 * s5;
    m.s0 += s3; m.s1 = fma(s3, b, m.s1);
    m.t0 += t5; m.t1 = fma(t5, b, m.t1);
  }
}

// The Taylor sums' range holds along every row of the element.
__device__ __forceinline__ bool regi_brief(const Elem& e, double kre, double kim)
{
  const double reach = regi_reach(e);
  return fabs(kre) * reach <= REGI_XMAX && fabs(kim) * reach <= REGI_YMAX;
}

// Adds the moments of row a, times its weight wr, to the 48 shape-function sums v[(8 q + 2 i + part) ld] of the
// quantities q = G, H, dG0, dG1, dH0, dH1, and to F, dF0, dF1.
__device__ __forceinline__ void regi_add(const RegiLine& y, const RegiRow& m, bool tri, int part, double a,
                                         const double* v0, const double* v1, double wr, double* v, int ld, double& F, double& dF0, double& dF1)
{
  const double C0 = dot3(y.C, v0), D0 = dot3(y.D, v0), C1 = dot3(y.C, v1), D1 = dot3(y.D, v1);
  const double P0 = dot3(y.P, v0), Q0 = dot3(y.Q, v0), P1 = dot3(y.P, v1), Q1 = dot3(y.Q, v1);
  // sums of f and f b of the integrands
  const cplx f0[6] = {m.g0, m.h0, m.a0 * P0 + m.a1 * Q0, m.a0 * P1 + m.a1 * Q1,
                      m.e0 * P0 + m.e1 * Q0 - (m.q0 * C0 + m.q1 * D0), m.e0 * P1 + m.e1 * Q1 - (m.q0 * C1 + m.q1 * D1)};
  const cplx f1[6] = {m.g1, m.h1, m.a1 * P0 + m.a2 * Q0, m.a1 * P1 + m.a2 * Q1,
                      m.e1 * P0 + m.e2 * Q0 - (m.q1 * C0 + m.q2 * D0), m.e1 * P1 + m.e2 * Q1 - (m.q1 * C1 + m.q2 * D1)};
  F += wr * m.F;
  dF0 += wr * (P0 * m.s0 + Q0 * m.s1 - (C0 * m.t0 + D0 * m.t1));
  dF1 += wr * (P1 * m.s0 + Q1 * m.s1 - (C1 * m.t0 + D1 * m.t1));
  double sa[4], sb[4];
  regi_shape(tri, part, a, sa, sb);
#pragma unroll
  for (int i = 0; i < 4; i++) {
    const double al = wr * sa[i], be = wr * sb[i];
#pragma unroll
    for (int c = 0; c < 6; c++) {
      double* p = v + (c * 8 + 2 * i) * ld;
      p[0] += al * f0[c].re + be * f1[c].re;
      p[ld] += al * f0[c].im + be * f1[c].im;
    }
  }
}

// load_elem where every lane has its own element: 32-byte loads where the records lie on such
// boundaries (a caller's array need not), a quarter of the sectors.
__device__ __forceinline__ void load_elem_wide(const double* __restrict__ geo, int id, Elem& e)
{
  if ((reinterpret_cast<uintptr_t>(geo) & 31) != 0) {
    load_elem(geo, id, e);
    return;
  }
  const double* g = geo + (size_t)id * GEO_STRIDE;
  double v[21];
#pragma unroll
  for (int i = 0; i < 20; i += 4)
    asm("ld.global.nc.v4.f64 {%0, %1, %2, %3}, [%4];" : "=d"(v[i]), "=d"(v[i + 1]), "=d"(v[i + 2]), "=d"(v[i + 3]) : "l"(g + i));
  v[20] = g[20];
  e.nn = (int)g[GEO_NN];
  const bool tri = e.nn == 3;
#pragma unroll
  for (int d = 0; d < 3; d++) {
#pragma unroll
    for (int c = 0; c < 4; c++) e.cr[d][c] = (tri && c == 3) ? 0.0 : v[4 * d + c];
#pragma unroll
    for (int c = 0; c < 3; c++) e.cw[d][c] = (tri && c > 0) ? 0.0 : v[12 + 3 * d + c];
  }
}

// WIDE: every matrix starts on 16 bytes (tested on the host: a test here costs the kernel 1 %).
template <bool WIDE>
__device__ __forceinline__ void reg_interior_warp(const AssembleArgs& A, int row, int s, int lane, double3* Fp,
                                                  long long fidx, unsigned* gh_list, unsigned* gh_count, unsigned gh_cap,
                                                  int* status, double* acc)
{
  const int t = row >> 2, tn = row & 3;
  const bool in = s < A.ne;
  int tnn;
  double rt[3], v0[3], v1[3];
  target_info(A.geo, A.sid, t, tn, rt, v0, v1, tnn);
  const bool blank = (tn == 3 && tnn == 3);  // a triangle's fourth row stays zero
  const int sd = A.sid[in ? s : 0];
  Elem e;
  load_elem_wide(A.geo, abs(sd), e);
  const bool tri = e.nn == 3;
  // What is not needed within a row waits in shared memory: the row's moments and linear forms take 100
  // registers, and spilled values would go through L2 (the sums leave L1 little room).
  double *my = acc + lane, *me = acc + 48 * REGI_LD + lane, *mu = acc + 48 * REGI_LD + 21 * 32;
#pragma unroll
  for (int i = 0; i < 12; i++) me[32 * i] = e.cr[i / 4][i % 4];
#pragma unroll
  for (int i = 0; i < 9; i++) me[32 * (12 + i)] = e.cw[i / 3][i % 3];
  if (lane < 3) { mu[lane] = rt[lane]; mu[3 + lane] = v0[lane]; mu[6 + lane] = v1[lane]; }
#pragma unroll
  for (int i = 0; i < 48; i++) my[i * REGI_LD] = 0.0;
  double F = 0.0, dF0 = 0.0, dF1 = 0.0;
  const bool none = blank || !in || s == t;
  const bool brief = __all_sync(0xffffffffu, none || regi_brief(e, A.kre, A.kim));
  // the warp's pairs take the largest of their rules: one loop count, and nodes from constant memory
  const double dx = e.cr[0][0] - rt[0], dy = e.cr[1][0] - rt[1], dz = e.cr[2][0] - rt[2];
  const int n = __reduce_max_sync(
      0xffffffffu, none ? RULE_NMIN : rule_order(e, dx * dx + dy * dy + dz * dz, fabs(A.kre) + 2.5 * fabs(A.kim)));
  const double *xn = c_xr + RULE_OFF(n), *wn = c_wr + RULE_OFF(n);
  const int nrow = none ? 0 : (tri ? 3 * n : n);
  __syncwarp();
#pragma unroll 1
  for (int ar = 0; ar < nrow; ar++) {
    const int part = (ar >= n) + (ar >= 2 * n), ia = ar - n * part;
    Elem er;
#pragma unroll
    for (int i = 0; i < 12; i++) er.cr[i / 4][i % 4] = me[32 * i];
#pragma unroll
    for (int i = 0; i < 9; i++) er.cw[i / 3][i % 3] = me[32 * (12 + i)];
    er.nn = tri ? 3 : 4;
    RegiLine y;
    regi_line(er, mu, part, xn[ia], y);
    RegiRow m;
    memset(&m, 0, sizeof m);
    if (brief) regi_row<true>(y, xn, wn, 0, n, tri, A.kre, A.kim, m);
    else regi_row<false>(y, xn, wn, 0, n, tri, A.kre, A.kim, m);
    regi_add(y, m, tri, part, xn[ia], mu + 3, mu + 6, wn[ia], my, REGI_LD, F, dF0, dF1);
  }
  // scalings of acci_finish; an element seen from its other side flips H and F
  double cg = EL_I_FP, ch = EL_I_FP, cf = EL_I_FP;
  if (tri) {
    const double V[3] = {me[32 * 12], me[32 * 15], me[32 * 18]}, c = 0.0625 * EL_SQ3 * EL_I_SPSQ3;
    cg = c * vnorm3(V);
    ch = cf = c;
  }
  if (sd < 0) { ch = -ch; cf = -cf; }
#pragma unroll
  for (int i = 0; i < 48; i++) {
    const int q = i >> 3;  // G, H, dG0, dG1, dH0, dH1
    my[i * REGI_LD] *= q == 0 ? cg : (q == 2 || q == 3) ? -cg : ch;
  }
  const double dFz = dF0 * cf, dFe = dF1 * cf;
  if (in && s != t && !blank) {
    if (needs_gh(dFz, dFe)) {  // its entries and F are written again from the list
      const unsigned slot = atomicAdd(gh_count, 1u);
      if (slot < gh_cap) gh_list[slot] = (unsigned)fidx;
      else record_status(status, -900);
    } else {
      Fp[fidx] = make_double3(F * cf, dFz, dFe);
    }
  }
  __syncwarp();
  const size_t N = (size_t)4 * A.ne;
  const int s0 = s - lane;
  double* const mat[6] = {A.G, A.H, A.dG, A.dG, A.dH, A.dH};
#pragma unroll 1
  for (int q = 0; q < 6; q++) {
    if (!mat[q]) continue;
    const size_t r = (q < 2) ? (size_t)row : (size_t)2 * row + (q & 1);
    cplx* out = (cplx*)mat[q] + r * N + (size_t)4 * s0;
#pragma unroll
    for (int c = 0; c < 4; c++) {
      const int k = c * 32 + lane, sl = k >> 2, i = k & 3;
      if (s0 + sl >= A.ne || (s0 + sl == t && !blank)) continue;
      const double* v = acc + (q * 8 + 2 * i) * REGI_LD + sl;
      if (WIDE) *reinterpret_cast<double2*>(out + k) = make_double2(v[0], v[REGI_LD]);
      else out[k] = mk(v[0], v[REGI_LD]);
    }
  }
  __syncwarp();
}

// Regular interior pairs of one chunk (rows r0 .. r0 + nr - 1).  One B200, the shell of 1,728 quads
// (11.9 M pairs, complex wave number): 38.5 -> 25.2 ms by the moments, -> 18.7 ms by fewer points for
// distant pairs (rule_order; 7 to 9 per direction for most), -> 13.5 ms with a warp per CTA, the elements
// in shared memory in place of spilled registers, and read by 32-byte loads.  FP64 pipe 60 % busy (45 % before),
// 168 registers, 12 CTAs a multiprocessor by registers and by shared memory.
#define REGI_BLOCKS 9  // 168 registers (three warps a partition); 16 with spilled registers took 18.7 ms
template <bool WIDE>
__global__ void __launch_bounds__(REGI_WARPS * 32, REGI_BLOCKS) k_reg_interior(AssembleArgs A, int r0, int nr, double3* Fp,
                                                                     unsigned* gh_list, unsigned* gh_count, unsigned gh_cap,
                                                                     int* status)
{
  extern __shared__ __align__(16) double regi_smem[];
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5, wpr = (A.ne + 31) >> 5;
  const long long w = (long long)blockIdx.x * REGI_WARPS + wib;
  if (w >= (long long)wpr * nr) return;  // uniform across the warp
  const int rr = (int)(w / wpr), s = (int)(w - (long long)rr * wpr) * 32 + lane;
  reg_interior_warp<WIDE>(A, r0 + rr, s, lane, Fp, (long long)rr * A.ne + s, gh_list, gh_count, gh_cap, status,
                    regi_smem + wib * REGI_SMEM);
}

// Near-singular interior pair w of the chunk starting at pair p0, 64 x 64 rule, by the whole CTA
// (GHI_THREADS threads): a thread takes half a row of 64 points at a time, by the regular rule's moments.
#define GHI_THREADS 128
__device__ __forceinline__ void gh_interior_pair(const AssembleArgs& A, long long p0, long long w, double3* Fp,
                                                 const double* xh, const double* wh, double (*red)[51])
{
  const PairIdx q = pair_of(p0 + w, A.ne);
  int tnn;
  double rt[3], v0[3], v1[3];
  target_info(A.geo, A.sid, q.t, q.tn, rt, v0, v1, tnn);
  const int sd = A.sid[q.s];
  Elem e;
  load_elem(A.geo, abs(sd), e);
  const bool tri = e.nn == 3;
  const bool brief = regi_brief(e, A.kre, A.kim);
  double v[51];
#pragma unroll
  for (int i = 0; i < 51; i++) v[i] = 0.0;
  const int items = tri ? 3 * 64 * 2 : 64 * 2;
#pragma unroll 1
  for (int it = threadIdx.x; it < items; it += GHI_THREADS) {
    const int half = it & 1, ar = it >> 1, part = ar >> 6, ia = ar & 63;
    RegiLine y;
    regi_line(e, rt, part, xh[ia], y);
    RegiRow m;
    memset(&m, 0, sizeof m);
    if (brief) regi_row<true>(y, xh, wh, 32 * half, 32 * half + 32, tri, A.kre, A.kim, m);
    else regi_row<false>(y, xh, wh, 32 * half, 32 * half + 32, tri, A.kre, A.kim, m);
    regi_add(y, m, tri, part, xh[ia], v0, v1, wh[ia], v, 1, v[48], v[49], v[50]);
  }
  warp_sum_arr<51>(v);
  const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (lane == 0)
    for (int i = 0; i < 51; i++) red[wid][i] = v[i];
  __syncthreads();
  if (threadIdx.x < 51) {
    double t = 0.0;
    for (int i = 0; i < GHI_THREADS / 32; i++) t += red[i][threadIdx.x];
    red[0][threadIdx.x] = t;
  }
  __syncthreads();
  if (wid == 0) {
    AccI a;
    const double* r = red[0];
    for (int i = 0; i < 4; i++) {
      a.G[i] = mk(r[2 * i], r[2 * i + 1]);
      a.H[i] = mk(r[8 + 2 * i], r[9 + 2 * i]);
      a.dG0[i] = mk(r[16 + 2 * i], r[17 + 2 * i]);
      a.dG1[i] = mk(r[24 + 2 * i], r[25 + 2 * i]);
      a.dH0[i] = mk(r[32 + 2 * i], r[33 + 2 * i]);
      a.dH1[i] = mk(r[40 + 2 * i], r[41 + 2 * i]);
    }
    a.F = r[48]; a.dF0 = r[49]; a.dF1 = r[50];
    cplx CC[9], dCz[9], dCe[9];
    acci_finish(e, a, sd < 0, CC, dCz, dCe);
    store_pair(A, q.row, q.s, CC, dCz, dCe, Fp, w, lane);
  }
  __syncthreads();
}

// Near-singular interior pairs of one chunk: one CTA per listed pair (at most gh_cap of them).
__global__ void __launch_bounds__(GHI_THREADS, 4) k_gh_interior(AssembleArgs A, long long p0, double3* Fp,
                                                                const unsigned* gh_list, const unsigned* gh_count,
                                                                unsigned gh_cap)
{
  __shared__ double red[GHI_THREADS / 32][51];
  __shared__ double xh[64], wh[64];
  const unsigned n = min(*gh_count, gh_cap);
  if (blockIdx.x >= n) return;
  if (threadIdx.x < 64) { xh[threadIdx.x] = c_xh[threadIdx.x]; wh[threadIdx.x] = c_wh[threadIdx.x]; }
  __syncthreads();
  for (unsigned it = blockIdx.x; it < n; it += gridDim.x) gh_interior_pair(A, p0, gh_list[it], Fp, xh, wh, red);
}

// ==========================================================================================
// Row sums (d3qd2_solve_bieq.c:222-236): F, dF/dtz, dF/dte over all s (regular pairs from the
// chunk scratch, the self pair from Fself), then H[row][4t+tn] += (did==0 ? 1 : 0) + F.
// One warp per row; lane-strided partial sums and a fixed-shape reduction (deterministic).
// fr: the row's F terms (ne of them, indexed by s).
__device__ __forceinline__ void rowsum_row(const AssembleArgs& A, int row, const double3* fr, const double3* Fself, int lane)
{
  int t = row >> 2, tn = row & 3;
  int at = abs(A.sid[t]);
  int tnn = (int)A.geo[(size_t)at * GEO_STRIDE + GEO_NN];
  if (tn == 3 && tnn == 3) return;
  double f0 = 0, f1 = 0, f2 = 0;
  for (int s = lane; s < A.ne; s += 32) {
    if (s == t) continue;
    double3 v = fr[s];
    f0 += v.x; f1 += v.y; f2 += v.z;
  }
  f0 = warp_sum(f0); f1 = warp_sum(f1); f2 = warp_sum(f2);
  if (lane == 0) {
    double3 sv = Fself[row];
    f0 += sv.x; f1 += sv.y; f2 += sv.z;
    double diag = (A.did == 0) ? 1.0 + f0 : f0;
    cplx* H = (cplx*)A.H;
    size_t N = (size_t)4 * A.ne;
    H[(size_t)row * N + 4 * (size_t)t + tn].re += diag;
    if (A.dF) {
      A.dF[3 * (size_t)row + 0] = diag;
      A.dF[3 * (size_t)row + 1] = f1;
      A.dF[3 * (size_t)row + 2] = f2;
    }
  }
}

__global__ void k_rowsum(AssembleArgs A, int row0, int nrows, const double3* Fp, const double3* Fself)
{
  int wr = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  int lane = threadIdx.x & 31;
  if (wr >= nrows) return;
  rowsum_row(A, row0 + wr, Fp + (size_t)wr * A.ne, Fself, lane);
}

// ==========================================================================================
// Self pairs of the periodic domain (q0_bil_dcoef_bd_vt2_cc_DV q0_bil_dcoef_v2_cc.c:292-301 and
// q0_lit_dcoef_bd_vt2_cc_DV q0_lit_dcoef_v2_cc.c:331-342).  One CTA per (t, tn); the point loop
// and the combination are self_per_points / self_per_combine (self.cuh).
#define SELF_THREADS 256
// Row `row` (= 4 t + tn) of the periodic domain, by the whole CTA (SELF_THREADS threads).
__device__ __forceinline__ void self_periodic_row(const AssembleArgs& A, const QPLattice& L, int row, double3* Fself,
                                                  int* status, double (*red)[24], int* serr)
{
  const int t = row >> 2, tn = row & 3;
  SelfInfo S;
  self_setup(A.geo, abs(A.sid[t]), tn, mk(0.0, 0.0), S);
  if (tn == 3 && S.e.nn == 3) return;
  double v[24];
  for (int i = 0; i < 24; i++) v[i] = 0.0;
  int err = self_per_points(S, L, c_xl, c_wl, c_xh, c_wh, threadIdx.x, blockDim.x, v);
  warp_sum_arr<24>(v);
  err = warp_min_i(err);
  int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (lane == 0) { for (int i = 0; i < 24; i++) red[wid][i] = v[i]; serr[wid] = err; }
  __syncthreads();
  if (wid != 0) return;
  for (int i = 0; i < 24; i++) v[i] = (lane < SELF_THREADS / 32) ? red[lane][i] : 0.0;
  warp_sum_arr<24>(v);
  int e3 = warp_min_i(lane < SELF_THREADS / 32 ? serr[lane] : 0);
  if (lane != 0) return;
  record_status(status, e3);
  cplx CC[9], dCz[9], dCe[9];
  self_per_combine(S, v, CC, dCz, dCe);
  store_pair(A, row, t, CC, dCz, dCe, Fself, row, -1);
}

__global__ void __launch_bounds__(SELF_THREADS, 2) k_self_periodic(AssembleArgs A, const __grid_constant__ QPLattice L,
                                                                   const SmoothPlan* plan, double3* Fself, int* status)
{
  if (plan && plan->on) return;
  __shared__ double red[SELF_THREADS / 32][24];
  __shared__ int serr[SELF_THREADS / 32];
  self_periodic_row(A, L, blockIdx.x, Fself, status, red, serr);
}

#include "assemble_smooth.cuh"

// ==========================================================================================
// Host side
static void gauleg_host(int n, double* x, double* w)
{
  // Gauss-Legendre nodes on [-1,1] by Newton iteration on P_n from the Chebyshev-like initial
  // guess, with the stop tolerance of the reference's gauleg (com_src/gauleg.c:3-36) so that the
  // tables agree bit for bit (near-singular pairs are sensitive to the last bits of the nodes).
  for (int i = 0; i < (n + 1) / 2; i++) {
    double z = cos(QP_PI * (i + 0.75) / (n + 0.5)), z1, pp;
    for (int it = 0; it < 100; it++) {
      double p1 = 1.0, p2 = 0.0;
      for (int j = 1; j <= n; j++) {
        double p3 = p2;
        p2 = p1;
        p1 = ((2.0 * j - 1.0) * z * p2 - (j - 1.0) * p3) / j;
      }
      pp = n * (z * p1 - p2) / (z * z - 1.0);
      z1 = z;
      z = z1 - p1 / pp;
      if (fabs(z - z1) <= 3.0e-16) break;
    }
    x[i] = -z;
    x[n - 1 - i] = z;
    w[i] = 2.0 / ((1.0 - z * z) * pp * pp);
    w[n - 1 - i] = w[i];
  }
}

static int g_tables_ready[64];

static int ensure_tables(void)
{
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 64 && g_tables_ready[dev]) return 0;
  double xl[12], wl[12], xh[64], wh[64];
  gauleg_host(12, xl, wl);
  gauleg_host(64, xh, wh);
  if (cudaMemcpyToSymbol(c_xl, xl, sizeof xl) != cudaSuccess) return -1;
  if (cudaMemcpyToSymbol(c_wl, wl, sizeof wl) != cudaSuccess) return -1;
  if (cudaMemcpyToSymbol(c_xh, xh, sizeof xh) != cudaSuccess) return -1;
  if (cudaMemcpyToSymbol(c_wh, wh, sizeof wh) != cudaSuccess) return -1;
  double xr[RULE_TAB], wr[RULE_TAB];
  for (int n = RULE_NMIN; n <= RULE_NMAX; n++) gauleg_host(n, xr + RULE_OFF(n), wr + RULE_OFF(n));
  if (cudaMemcpyToSymbol(c_xr, xr, sizeof xr) != cudaSuccess) return -1;
  if (cudaMemcpyToSymbol(c_wr, wr, sizeof wr) != cudaSuccess) return -1;
  double xs[SELF_NLOG], ws[SELF_NLOG];
  gauleg_host(SELF_NLOG, xs, ws);
  if (cudaMemcpyToSymbol(c_xs, xs, sizeof xs) != cudaSuccess) return -1;
  if (cudaMemcpyToSymbol(c_ws, ws, sizeof ws) != cudaSuccess) return -1;
  // k_reg_periodic keeps ~80 KB of shared memory per block (dynamic, above the 48 KB static
  // limit): allow it, and ask for the largest carve-out so the L1 split does not cut occupancy
  if (cudaFuncSetAttribute(k_reg_periodic, cudaFuncAttributePreferredSharedMemoryCarveout,
                           (int)cudaSharedmemCarveoutMaxShared) != cudaSuccess ||
      cudaFuncSetAttribute(k_reg_periodic, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)REGP_SMEM_BYTES) !=
          cudaSuccess ||
      cudaFuncSetAttribute(k_reg_smooth, cudaFuncAttributePreferredSharedMemoryCarveout,
                           (int)cudaSharedmemCarveoutMaxShared) != cudaSuccess ||
      cudaFuncSetAttribute(k_reg_smooth, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int)(SMT_WARPS * sizeof(SmoothWarp))) != cudaSuccess ||
      cudaFuncSetAttribute(k_smooth_spectral, cudaFuncAttributeMaxDynamicSharedMemorySize, SMT_SPEC_SMEM) != cudaSuccess)
    return -1;
  for (auto reg : {k_reg_interior<true>, k_reg_interior<false>})
    if (cudaFuncSetAttribute(reg, cudaFuncAttributePreferredSharedMemoryCarveout, (int)cudaSharedmemCarveoutMaxShared) !=
            cudaSuccess ||
        cudaFuncSetAttribute(reg, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)REGI_SMEM_BYTES) != cudaSuccess)
      return -1;
  if (dev < 64) g_tables_ready[dev] = 1;
  return 0;
}

extern "C" void bem3_gauss_legendre(int n, double* x, double* w) { gauleg_host(n, x, w); }

// Scratch layout of bem3_assemble_run for a chunk of `rows` rows, each part starting on a 256-byte
// boundary: self-pair F sums (4 ne double3), the work-list counters (256 B), the chunk's per-pair F
// terms (rows * ne double3), the near-singular work list (rows * ne / 8 + 4096 u32), and for a table of
// `cap` coefficients (periodic domains; 0: none) the plan, the list of in-plane pairs (rows * ne u32),
// the coefficients and the samples.
static inline size_t round256(size_t b) { return (b + 255) & ~(size_t)255; }
struct ScratchLayout {
  size_t fself, counters, fp, gh_list, plan, ip_list, tab, smp, end;
  unsigned gh_cap;
};
static ScratchLayout scratch_layout(int ne, int rows, long long cap)
{
  ScratchLayout l;
  const size_t np = (size_t)rows * ne;
  l.gh_cap = (unsigned)(np / 8 + 4096);
  l.fself = 0;
  l.counters = round256((size_t)4 * ne * sizeof(double3));
  l.fp = l.counters + 256;
  l.gh_list = l.fp + round256(np * sizeof(double3));
  l.plan = l.gh_list + round256((size_t)l.gh_cap * sizeof(unsigned));
  l.ip_list = l.plan + (cap ? round256(sizeof(SmoothPlan)) : 0);
  l.tab = l.ip_list + (cap ? round256(np * sizeof(unsigned)) : 0);
  l.smp = l.tab + round256((size_t)cap * sizeof(cplx));
  l.end = l.smp + round256((size_t)cap * 2 * sizeof(cplx));
  return l;
}
size_t bem3_scratch_bytes(int ne, int rows, long long cap) { return scratch_layout(ne, rows, cap).end; }

// Runs the whole domain on `stream` using caller-provided scratch (see bem3_scratch_bytes).
// Returns 0, or a negative code (see bem3_qd2_b200.h).
// Adds a chunk's near-singular count to the domain's total (no host round trip per chunk).
__global__ void k_acc_count(const unsigned* __restrict__ cnt, unsigned long long* __restrict__ total)
{
  *total += *cnt;
}

int bem3_assemble_run(const AssembleArgs& A, const QPLattice* L, const SmoothLat* S, void* scratch, size_t scratch_bytes,
                      int rows_per_chunk, long long cap, int* d_status, cudaStream_t st, AssembleStats* stats,
                      const ChunkHook* hook)
{
  if (ensure_tables() != 0) return BEM3_ERR_CUDA;
  const int ne = A.ne;
  const int nrows = 4 * ne;
  if (rows_per_chunk <= 0 || rows_per_chunk > nrows) rows_per_chunk = nrows;
  SmoothArgs M;
  memset(&M, 0, sizeof M);
  if (A.periodic && S) M.S = *S;
  if (!M.S.ok) cap = 0;
  const ScratchLayout lay = scratch_layout(ne, rows_per_chunk, cap);
  if (lay.end > scratch_bytes) return BEM3_ERR_SCRATCH;  // every part below ends inside the scratch
  char* base = (char*)scratch;
  double3* Fself = (double3*)(base + lay.fself);
  unsigned* gh_count = (unsigned*)(base + lay.counters);                          // this chunk's list length
  unsigned long long* gh_total = (unsigned long long*)(base + lay.counters + 8);  // the domain's total
  double3* Fp = (double3*)(base + lay.fp);
  unsigned* gh_list = (unsigned*)(base + lay.gh_list);
  const unsigned gh_cap = lay.gh_cap;
  // tabulated pairs: their near-singular list fills gh_list, the in-plane pairs' (ip_list) the same
  // way after them; both lists' counters
  unsigned* smt_count = (unsigned*)(base + lay.counters + 16);
  unsigned* ip_count = (unsigned*)(base + lay.counters + 20);
  unsigned* ip_list = (unsigned*)(base + lay.ip_list);
  if (cap) {
    M.plan = (SmoothPlan*)(base + lay.plan);
    M.tab = (cplx*)(base + lay.tab);
    M.smp = (cplx*)(base + lay.smp);
    M.cap = cap;
  }

  const size_t N = (size_t)nrows;
  if (A.periodic) {  // its kernels skip the triangles' fourth rows and the derivatives (all zero)
    if (cudaMemsetAsync(A.G, 0, N * N * 16, st) != cudaSuccess) return BEM3_ERR_CUDA;
    if (cudaMemsetAsync(A.H, 0, N * N * 16, st) != cudaSuccess) return BEM3_ERR_CUDA;
    if (A.dG && cudaMemsetAsync(A.dG, 0, 2 * N * N * 16, st) != cudaSuccess) return BEM3_ERR_CUDA;
    if (A.dH && cudaMemsetAsync(A.dH, 0, 2 * N * N * 16, st) != cudaSuccess) return BEM3_ERR_CUDA;
  }
  if (A.dF && cudaMemsetAsync(A.dF, 0, N * 3 * sizeof(double), st) != cudaSuccess) return BEM3_ERR_CUDA;
  cudaMemsetAsync(Fself, 0, N * sizeof(double3), st);
  cudaMemsetAsync(gh_total, 0, sizeof(unsigned long long), st);

  int launches = 0;
  cudaEvent_t ev0 = nullptr, ev1 = nullptr;
  const bool timing = stats && stats->time_kernels;
  if (timing) { cudaEventCreate(&ev0); cudaEventCreate(&ev1); }
  // profiling only: the duration of the kernels launched since tic() goes to class_ms[cls]
  auto tic = [&]() { if (timing) cudaEventRecord(ev0, st); };
  auto toc = [&](int cls) -> float {
    float ms = 0.f;
    if (timing) {
      cudaEventRecord(ev1, st);
      cudaEventSynchronize(ev1);
      cudaEventElapsedTime(&ms, ev0, ev1);
      stats->class_ms[cls] += ms;
    }
    return ms;
  };
  // the table of the smooth remainder
  if (M.plan) {
    tic();
    k_smooth_plan<<<1, SMT_PLAN_THREADS, 0, st>>>(A, *L, M);
    k_smooth_spectral<<<148 * 4, SMT_SPEC_THREADS, smooth_spec_smem(M.S), st>>>(*L, M);
    k_smooth_project<<<148 * 8, SMT_PROJ_THREADS, 0, st>>>(*L, M);
    toc(1);
    launches += 3;
    if (timing && cudaMemcpy(&stats->table_on, &M.plan->on, sizeof(int), cudaMemcpyDeviceToHost) != cudaSuccess)
      return BEM3_ERR_CUDA;
  }
  // self pairs
  tic();
  if (A.periodic) {
    if (M.plan) { k_self_smooth<<<nrows, SELF_THREADS, 0, st>>>(A, *L, M, Fself); launches++; }
    k_self_periodic<<<nrows, SELF_THREADS, 0, st>>>(A, *L, M.plan, Fself, d_status);
  } else {
    bem3_launch_self_interior(A, Fself, d_status, st);
  }
  toc(0);
  launches++;

  for (int r0 = 0; r0 < nrows; r0 += rows_per_chunk) {
    int nr = (r0 + rows_per_chunk <= nrows) ? rows_per_chunk : nrows - r0;
    long long p0 = (long long)r0 * ne, np = (long long)nr * ne;
    cudaMemsetAsync(gh_count, 0, sizeof(unsigned), st);
    if (A.periodic) {
      const long long units = (np + REGP_PAIRS - 1) / REGP_PAIRS;
      // without a table every pair has its warp; with one, a resident grid strides over what it left
      const long long want = (units * 32 + 255) / 256;
      const unsigned blocks = (unsigned)((M.plan && want > 148 * REGP_MIN_BLOCKS) ? 148 * REGP_MIN_BLOCKS : want);
      tic();
      if (M.plan) {
        cudaMemsetAsync(smt_count, 0, 2 * sizeof(unsigned), st);
        const long long su = (long long)((ne + SMT_PAIRS - 1) / SMT_PAIRS) * nr;
        k_reg_smooth<<<(unsigned)((su + SMT_WARPS - 1) / SMT_WARPS), SMT_WARPS * 32, SMT_WARPS * sizeof(SmoothWarp), st>>>(
            A, *L, M, r0, nr, Fp, gh_list, smt_count, gh_cap, ip_list, ip_count, d_status);
        launches++;
      }
      const float sms = toc(1);
      if (timing && M.plan) {
        unsigned left = 0;
        if (cudaMemcpy(&left, ip_count, sizeof left, cudaMemcpyDeviceToHost) != cudaSuccess) return BEM3_ERR_CUDA;
        stats->reg_smooth_ms += sms;
        stats->plane_pairs += left;
      }
      tic();
      if (M.plan) {
        k_gh_smooth<<<148 * 4, 256, 0, st>>>(A, *L, M, p0, Fp, gh_list, smt_count, gh_cap);
        k_acc_count<<<1, 1, 0, st>>>(smt_count, gh_total);
        launches += 2;
      }
      toc(2);
      tic();
      k_reg_periodic<<<blocks, 256, REGP_SMEM_BYTES, st>>>(A, *L, M.plan, ip_list, ip_count, p0, np, Fp, gh_list, gh_count,
                                                           gh_cap, d_status);
      const float ms = toc(1);
      if (timing) {
        stats->reg_periodic_ms += ms;
        stats->reg_periodic_launches++;
      }
      tic();
      k_gh_periodic<<<148 * 4, 256, 0, st>>>(A, *L, p0, Fp, gh_list, gh_count, gh_cap, d_status);
      toc(2);
    } else {
      const long long warps = (long long)((ne + 31) / 32) * nr;
      tic();
      const auto reg = wide_outputs(A) ? k_reg_interior<true> : k_reg_interior<false>;
      reg<<<(unsigned)((warps + REGI_WARPS - 1) / REGI_WARPS), REGI_WARPS * 32, REGI_SMEM_BYTES, st>>>(
          A, r0, nr, Fp, gh_list, gh_count, gh_cap, d_status);
      toc(1);
      tic();
      k_gh_interior<<<148 * 8, GHI_THREADS, 0, st>>>(A, p0, Fp, gh_list, gh_count, gh_cap);
      toc(2);
    }
    tic();
    k_rowsum<<<(nr * 32 + 255) / 256, 256, 0, st>>>(A, r0, nr, Fp, Fself);
    toc(3);
    k_acc_count<<<1, 1, 0, st>>>(gh_count, gh_total);
    launches += 4;
    if (hook) hook->fn(hook->user, r0, nr, st);
  }
  if (timing) { cudaEventDestroy(ev0); cudaEventDestroy(ev1); }
  if (stats) {
    stats->launches += launches;
    stats->d_gh_total = gh_total;
  }
  if (cudaGetLastError() != cudaSuccess) return BEM3_ERR_CUDA;
  return 0;
}
