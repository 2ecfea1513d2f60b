// batch.cu -- the coefficient matrices of many domains of many instances (meshes, wavelengths,
// incidence angles, lattices) assembled together: one launch per pair class for the whole batch,
// fed from device work lists, replayed as one CUDA graph.
//
// The reference assembles one domain at a time (create_cmatrix_domain,
// d3qd2_src/d3qd2_solve_bieq.c:165-256), and so does bem3_assemble_domain_dev.  A batch of
// instances of uneven size run that way leaves the GPU partly idle at the end of every launch
// and launches (self, regular, near-singular, row sums) per domain.  Here:
//
//   descriptor table  BatchDomain[nd] in device memory: the domain's AssembleArgs, its own
//                     QPLattice (Bloch wave vector, Ewald split parameter veps0, propagating
//                     orders), its scratch (per-pair F terms, near-singular work list,
//                     status word) and, for periodic domains, the plan and table of the smooth
//                     remainder (assemble_smooth.cuh), which every run makes anew;
//   work segments     per pair class, the cumulative work of the domains of that class
//                     (rows, pairs or pair units); a launch maps its global work index to
//                     (domain, local index) by binary search over them;
//   persistent kernel k_batch_reg_periodic, the pairs summed point by point (domains without a
//                     table, and the pairs in one plane that a table leaves): every warp takes
//                     `grab` units of REGP_PAIRS pairs at a time from one device counter until they
//                     are exhausted, whatever domain they belong to;
//   graph             reset, zero, then two branches -- periodic (tables, self, regular,
//                     near-singular) and interior (self, regular, near-singular) -- joined before the
//                     row sums.
//
// Every pair is computed by the same device functions, in the same order of operations, as in
// the one-domain kernels (assemble.cu), so a domain's matrices do not depend on what else is in
// the batch.  Measured on a B200, four two-layer problems of 192 quads with creation and wait: 218 ms
// with point-by-point periodic sums, 25.5 ms with the tables.
#include <cuda_runtime.h>
#include <string.h>

#include <algorithm>
#include <vector>

#include "bem3_internal.h"

struct BatchDomain {
  AssembleArgs A;
  QPLattice L;         // periodic domains only; L.prop points into the batch's list buffer
  double3* Fp;         // [4 ne * ne] per-pair F terms (the domain is one chunk)
  double3* Fself;      // [4 ne]
  unsigned* gh_list;   // [gh_cap] near-singular pairs (pair index within the domain)
  unsigned* gh_count;  // entries appended (may exceed gh_cap: then status -900)
  unsigned gh_cap;
  int* status;         // the domain's status word (first error code)
  SmoothArgs M;        // periodic domains: plan and table (plan == nullptr: none)
  unsigned* ip_list;   // [4 ne * ne] pairs in one plane, left to the point-by-point sums
  unsigned* smt_list;  // [gh_cap] near-singular pairs of the tabulated ones
  unsigned* smt_count; // entries of smt_list, then of ip_list; then whether the domain has a table (its plan's `on`)
};

// Cumulative work of the domains of one class: base[0] = 0, base[n] = total, domain dom[i]
// holds work [base[i], base[i + 1]).
struct BatchSeg {
  const long long* base;
  const int* dom;
  int n;
};

__device__ __forceinline__ int seg_find(const BatchSeg& S, long long x)
{
  int lo = 0, hi = S.n;
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (S.base[mid] <= x) lo = mid;
    else hi = mid;
  }
  return lo;
}

// Counters of a run: [0] regular periodic units taken.  Status words and work-list counters of
// every domain are cleared too.
__global__ void k_batch_reset(BatchDomain* D, int nd, unsigned long long* next)
{
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i == 0) next[0] = 0ull;
  if (i < nd) {
    *D[i].gh_count = 0u;
    if (D[i].smt_count) D[i].smt_count[0] = D[i].smt_count[1] = D[i].smt_count[2] = 0u;
    *D[i].status = 0;
  }
}

// Zeroes every output of domain blockIdx.y (rows of triangles with tn = 3 stay zero, as in the
// reference) and its self-pair F slots.
__global__ void k_batch_zero(const BatchDomain* __restrict__ D)
{
  const BatchDomain& d = D[blockIdx.y];
  const size_t N = (size_t)4 * d.A.ne;
  const size_t nn = N * N;
  const size_t stride = (size_t)gridDim.x * blockDim.x;
  const size_t i0 = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  auto zero = [&](double* m, size_t n) {  // n complex entries
    if (!m) return;
    if (wide_cplx(m)) {
      for (size_t i = i0; i < n; i += stride) ((double2*)m)[i] = make_double2(0.0, 0.0);
    } else {
      for (size_t i = i0; i < 2 * n; i += stride) m[i] = 0.0;
    }
  };
  if (d.A.periodic) {  // the interior kernels write every entry
    zero(d.A.G, nn);
    zero(d.A.H, nn);
    zero(d.A.dG, 2 * nn);
    zero(d.A.dH, 2 * nn);
  }
  if (d.A.dF) for (size_t i = i0; i < 3 * N; i += stride) d.A.dF[i] = 0.0;
  for (size_t i = i0; i < N; i += stride) d.Fself[i] = make_double3(0.0, 0.0, 0.0);
}

// Tables of the periodic domains dom[blockIdx.y].  The tables of a batch share one pool of memory: the domains go
// through it in groups, plan to near-singular pairs, group after group (bem3_batch_create).
__global__ void __launch_bounds__(SMT_PLAN_THREADS) k_batch_smooth_plan(const BatchDomain* __restrict__ D,
                                                                        const int* __restrict__ dom)
{
  const BatchDomain& d = D[dom[blockIdx.x]];
  if (!d.M.plan) return;
  smooth_plan_block(d.A, d.L, d.M);
  __syncthreads();
  if (threadIdx.x == 0) d.smt_count[2] = (unsigned)d.M.plan->on;  // the plan's memory is another domain's later
}
__global__ void __launch_bounds__(SMT_SPEC_THREADS) k_batch_smooth_spectral(const BatchDomain* __restrict__ D,
                                                                            const int* __restrict__ dom)
{
  extern __shared__ __align__(16) unsigned char spec_smem[];
  const BatchDomain& d = D[dom[blockIdx.y]];
  if (d.M.plan) smooth_spectral_block(d.L, d.M, blockIdx.x, gridDim.x, spec_smem);
}
__global__ void __launch_bounds__(SMT_PROJ_THREADS) k_batch_smooth_project(const BatchDomain* __restrict__ D,
                                                                           const int* __restrict__ dom)
{
  const BatchDomain& d = D[dom[blockIdx.y]];
  if (d.M.plan) smooth_project_block(d.L, d.M, blockIdx.x, gridDim.x);
}

__device__ __forceinline__ bool batch_smooth(const BatchDomain& d) { return d.smt_count && d.smt_count[2] != 0u; }

__global__ void __launch_bounds__(SELF_THREADS, 2) k_batch_self_periodic(const BatchDomain* __restrict__ D, BatchSeg S)
{
  __shared__ double red[SELF_THREADS / 32][24];
  __shared__ int serr[SELF_THREADS / 32];
  const long long g = blockIdx.x;
  const int i = seg_find(S, g);
  const BatchDomain& d = D[S.dom[i]];
  if (batch_smooth(d)) return;
  self_periodic_row(d.A, d.L, (int)(g - S.base[i]), d.Fself, d.status, red, serr);
}

// Self pairs of the rows first, first + 1, ... of all periodic domains' rows.
__global__ void __launch_bounds__(SELF_THREADS, 2) k_batch_self_smooth(const BatchDomain* __restrict__ D, BatchSeg S,
                                                                       long long first)
{
  __shared__ double red[SELF_THREADS / 32][24];
  __shared__ double xl[12], wl[12], xh[64], wh[64];
  const long long g = first + blockIdx.x;
  const int i = seg_find(S, g);
  const BatchDomain& d = D[S.dom[i]];
  if (!batch_smooth(d)) return;
  if (threadIdx.x < 12) { xl[threadIdx.x] = c_xl[threadIdx.x]; wl[threadIdx.x] = c_wl[threadIdx.x]; }
  if (threadIdx.x < 64) { xh[threadIdx.x] = c_xh[threadIdx.x]; wh[threadIdx.x] = c_wh[threadIdx.x]; }
  __syncthreads();
  self_smooth_row(d.A, d.L, *d.M.plan, d.M.tab, (int)(g - S.base[i]), d.Fself, red, xl, wl, xh, wh);
}

// Tabulated regular pairs: S counts units of SMT_PAIRS sources (reg_smooth_unit), one warp each, from unit `first`
// to before `end`.
__global__ void __launch_bounds__(SMT_WARPS * 32, SMT_BLOCKS) k_batch_reg_smooth(const BatchDomain* __restrict__ D, BatchSeg S,
                                                                                 long long first, long long end)
{
  extern __shared__ __align__(16) unsigned char smt_smem[];
  __shared__ double xr[RULE_TAB], wr[RULE_TAB];
  for (int i = threadIdx.x; i < RULE_TAB; i += SMT_WARPS * 32) { xr[i] = c_xr[i]; wr[i] = c_wr[i]; }
  __syncthreads();
  const int wib = threadIdx.x >> 5;
  const long long u = first + (long long)blockIdx.x * SMT_WARPS + wib;
  if (u >= end) return;  // uniform across the warp
  const int i = seg_find(S, u);
  const BatchDomain& d = D[S.dom[i]];
  if (!batch_smooth(d)) return;
  reg_smooth_unit(d.A, d.L, d.M, 0, u - S.base[i], d.Fp, d.smt_list, d.smt_count, d.gh_cap, d.ip_list, d.smt_count + 1,
                  d.status, reinterpret_cast<SmoothWarp*>(smt_smem)[wib], xr, wr, threadIdx.x & 31);
}

__global__ void __launch_bounds__(SI_THREADS, 2) k_batch_self_interior(const BatchDomain* __restrict__ D, BatchSeg S)
{
  __shared__ double red[SI_NW * SELF_NV];
  __shared__ double res[4][SELF_NV];
  const long long g = blockIdx.x;
  const int i = seg_find(S, g);
  const BatchDomain& d = D[S.dom[i]];
  self_interior_row(d.A, (int)(g - S.base[i]), d.Fself, red, res);
}

// Persistent: gridDim.x CTAs of 8 warps; a warp takes `grab` units (REGP_PAIRS pairs each) per
// atomic on next[0] and runs them, until the units of all periodic domains are taken.
__global__ void __launch_bounds__(256, REGP_MIN_BLOCKS) k_batch_reg_periodic(const BatchDomain* __restrict__ D, BatchSeg S,
                                                                             int grab, unsigned long long* next)
{
  extern __shared__ __align__(16) unsigned char regp_smem[];  // REGP_SMEM_BYTES
  RegWarp(*sw)[REGP_PAIRS] = reinterpret_cast<RegWarp(*)[REGP_PAIRS]>(regp_smem);
  AccP(*sacc)[256] = reinterpret_cast<AccP(*)[256]>(regp_smem + sizeof(RegWarp) * 8 * REGP_PAIRS);
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  const long long total = S.base[S.n];
  for (;;) {
    unsigned long long u0 = 0ull;
    if (lane == 0) u0 = atomicAdd(next, (unsigned long long)grab);
    u0 = __shfl_sync(0xffffffffu, u0, 0);
    if ((long long)u0 >= total) break;
    const long long uend = min(total, (long long)u0 + grab);
    for (long long u = (long long)u0; u < uend; u++) {
      const int i = seg_find(S, u);
      const BatchDomain& d = D[S.dom[i]];
      const bool on = batch_smooth(d);  // then only the pairs in one plane are left
      const long long np = on ? (long long)d.smt_count[1] : 4LL * d.A.ne * d.A.ne;
      const long long first = (u - S.base[i]) * REGP_PAIRS;
      if (first >= np) continue;
      reg_periodic_unit(d.A, d.L, 0, np, first, on ? d.ip_list : nullptr, d.Fp, d.gh_list, d.gh_count, d.gh_cap, d.status,
                        sw[wib], sacc, lane);
    }
  }
}

// Regular interior pairs: S counts warps, each 32 sources of a row (reg_interior_warp).
template <bool WIDE>
__global__ void __launch_bounds__(REGI_WARPS * 32, REGI_BLOCKS) k_batch_reg_interior(const BatchDomain* __restrict__ D, BatchSeg S)
{
  extern __shared__ __align__(16) double regi_smem[];
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  const long long w = (long long)blockIdx.x * REGI_WARPS + wib;
  if (w >= S.base[S.n]) return;  // uniform across the warp
  const int i = seg_find(S, w);
  const BatchDomain& d = D[S.dom[i]];
  const int wpr = (d.A.ne + 31) >> 5;
  const long long u = w - S.base[i];
  const int row = (int)(u / wpr), s = (int)(u - (long long)row * wpr) * 32 + lane;
  reg_interior_warp<WIDE>(d.A, row, s, lane, d.Fp, (long long)row * d.A.ne + s, d.gh_list, d.gh_count, d.gh_cap, d.status,
                    regi_smem + wib * REGI_SMEM);
}

// Near-singular pairs: the domains' lists in turn, CTAs striding over each.
__global__ void __launch_bounds__(256, 2) k_batch_gh_periodic(const BatchDomain* __restrict__ D, const int* __restrict__ dom, int n)
{
  __shared__ double red[8][19];
  __shared__ int serr[8];
  for (int i = 0; i < n; i++) {
    const BatchDomain& d = D[dom[i]];
    const unsigned cnt = min(*d.gh_count, d.gh_cap);
    for (unsigned it = blockIdx.x; it < cnt; it += gridDim.x) gh_periodic_pair(d.A, d.L, 0, d.gh_list[it], d.Fp, d.status, red, serr);
  }
}

__global__ void __launch_bounds__(256, 2) k_batch_gh_smooth(const BatchDomain* __restrict__ D, const int* __restrict__ dom, int n)
{
  __shared__ double red[8][19];
  __shared__ double xh[64], wh[64];
  if (threadIdx.x < 64) { xh[threadIdx.x] = c_xh[threadIdx.x]; wh[threadIdx.x] = c_wh[threadIdx.x]; }
  __syncthreads();
  for (int i = 0; i < n; i++) {
    const BatchDomain& d = D[dom[i]];
    if (!batch_smooth(d)) continue;
    const unsigned cnt = min(d.smt_count[0], d.gh_cap);
    for (unsigned it = blockIdx.x; it < cnt; it += gridDim.x)
      gh_smooth_pair(d.A, d.L, *d.M.plan, d.M.tab, 0, d.smt_list[it], d.Fp, red, xh, wh);
  }
}

__global__ void __launch_bounds__(GHI_THREADS, 4) k_batch_gh_interior(const BatchDomain* __restrict__ D,
                                                                      const int* __restrict__ dom, int n)
{
  __shared__ double red[GHI_THREADS / 32][51];
  __shared__ double xh[64], wh[64];
  if (threadIdx.x < 64) { xh[threadIdx.x] = c_xh[threadIdx.x]; wh[threadIdx.x] = c_wh[threadIdx.x]; }
  __syncthreads();
  for (int i = 0; i < n; i++) {
    const BatchDomain& d = D[dom[i]];
    const unsigned cnt = min(*d.gh_count, d.gh_cap);
    for (unsigned it = blockIdx.x; it < cnt; it += gridDim.x) gh_interior_pair(d.A, 0, d.gh_list[it], d.Fp, xh, wh, red);
  }
}

// Row sums of every domain: one warp per row.
__global__ void k_batch_rowsum(const BatchDomain* __restrict__ D, BatchSeg S)
{
  const long long g = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (g >= S.base[S.n]) return;
  const int i = seg_find(S, g);
  const BatchDomain& d = D[S.dom[i]];
  const int row = (int)(g - S.base[i]);
  rowsum_row(d.A, row, d.Fp + (size_t)row * d.A.ne, d.Fself, threadIdx.x & 31);
}

// ------------------------------------------------------------------------------------------
// Host side
struct bem3_batch_s {
  int dev = 0;
  int nd = 0;
  void* mem = nullptr;  // one device allocation: table, segments, lists, scratch
  size_t bytes = 0;
  BatchDomain* dD = nullptr;
  int* dstatus = nullptr;
  cudaGraph_t graph = nullptr;
  cudaGraphExec_t exec = nullptr;
  int launches = 0;
};

namespace {

struct SegHost {
  std::vector<long long> base{0};
  std::vector<int> dom;
  void add(int d, long long work)
  {
    if (work <= 0) return;
    dom.push_back(d);
    base.push_back(base.back() + work);
  }
  long long total() const { return base.back(); }
  int n() const { return (int)dom.size(); }
};

// Bump allocator over the batch's single device allocation (256-byte aligned pieces).
struct Layout {
  size_t off = 0;
  size_t take(size_t bytes)
  {
    const size_t at = off;
    off += (bytes + 255) & ~(size_t)255;
    return at;
  }
};

void batch_free(bem3_batch b)
{
  if (!b) return;
  if (b->exec) cudaGraphExecDestroy(b->exec);
  if (b->graph) cudaGraphDestroy(b->graph);
  if (b->mem) cudaFree(b->mem);
  delete b;
}

}  // namespace

namespace {

// The pool that the batch's tables share: at most this many bytes, where one domain does not need more.
#define BATCH_POOL_BYTES ((size_t)2 << 30)

// A periodic domain's share of the pool, from its first byte: plan, table, samples, near-singular list.
struct PoolPart {
  size_t tab, smp, list, end;
};
PoolPart pool_part(long long cap, unsigned gh_cap)
{
  PoolPart p;
  p.tab = round256(sizeof(SmoothPlan));
  p.smp = p.tab + round256(sizeof(cplx) * (size_t)cap);
  p.list = p.smp + round256(sizeof(cplx) * 2 * (size_t)cap);
  p.end = p.list + round256(sizeof(unsigned) * (size_t)gh_cap);
  return p;
}

long long batch_table_room(const QPLattice& L, const SmoothLat& S, int ne)
{
  return smooth_capacity(L, S, ne, 4.0 * (double)ne * ne, 144.0, 0.0);
}

}  // namespace

extern "C" size_t bem3_batch_scratch_bytes(const bem3_batch_domain* doms, int n)
{
  if (!doms || n <= 0) return 0;
  size_t total = 0, pool = 0, largest = 0;
  for (int i = 0; i < n; i++) {
    const size_t ne = (size_t)(doms[i].Ne_d > 0 ? doms[i].Ne_d : 0);
    const size_t np = 4 * ne * ne;
    total += ((np * sizeof(double3) + 255) & ~(size_t)255) + ((4 * ne * sizeof(double3) + 255) & ~(size_t)255) +
             (((np / 8 + 4096) * sizeof(unsigned) + 255) & ~(size_t)255) + 256;
    if (doms[i].periodic) {
      total += (sizeof(QPProp) * QP_PROP_CAP + 255) & ~(size_t)255;
      QPLattice L;
      SmoothLat S;
      memset(&L, 0, sizeof L);
      if (ne == 0 || lattice_from(&doms[i].qd, &L) != 0) continue;  // refused by bem3_batch_create
      smooth_lattice(L, S);
      const long long cap = batch_table_room(L, S, (int)ne);
      if (cap == 0) continue;
      total += round256(np * sizeof(unsigned)) + 256;
      const size_t part = pool_part(cap, (unsigned)(np / 8 + 4096)).end;
      pool += part;
      largest = std::max(largest, part);
    }
  }
  total += std::min(pool, std::max(largest, BATCH_POOL_BYTES));
  // table, status words and segments
  total += (((sizeof(BatchDomain) + 2 * sizeof(long long) + 5 * sizeof(int)) * (size_t)n + 8 * sizeof(long long)) * 5 +
            255) & ~(size_t)255;
  return total + 4096;
}

extern "C" int bem3_batch_create(const bem3_batch_domain* doms, int n, const bem3_batch_tuning* tune, bem3_batch* out)
{
  if (!out) return BEM3_ERR_ARG;
  *out = nullptr;
  if (!doms || n <= 0 || n > 65535) return BEM3_ERR_ARG;  // the zero kernel's grid has one row per domain
  bem3_batch_tuning T = {8, REGP_MIN_BLOCKS, 4};
  if (tune) T = *tune;
  if (T.grab_units < 1 || T.grab_units > 4096 || T.regp_blocks_per_sm < 1 || T.regp_blocks_per_sm > REGP_MIN_BLOCKS ||
      T.gh_blocks_per_sm < 1 || T.gh_blocks_per_sm > 16)
    return BEM3_ERR_ARG;
  for (int i = 0; i < n; i++) {
    const bem3_batch_domain& d = doms[i];
    if (!d.geo || !d.sid || d.Ne <= 0 || d.Ne_d <= 0 || d.Ne_d > 2 * d.Ne || !d.G || !d.H) return BEM3_ERR_ARG;
    // pair indices of a domain's work list are 32-bit
    if (4.0 * d.Ne_d * (double)d.Ne_d >= 4294967295.0) return BEM3_ERR_ARG;
  }
  if (ensure_tables() != 0) return BEM3_ERR_CUDA;
  if (cudaFuncSetAttribute(k_batch_reg_periodic, cudaFuncAttributePreferredSharedMemoryCarveout,
                           (int)cudaSharedmemCarveoutMaxShared) != cudaSuccess ||
      cudaFuncSetAttribute(k_batch_reg_periodic, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)REGP_SMEM_BYTES) !=
          cudaSuccess ||
      cudaFuncSetAttribute(k_batch_reg_smooth, cudaFuncAttributePreferredSharedMemoryCarveout,
                           (int)cudaSharedmemCarveoutMaxShared) != cudaSuccess ||
      cudaFuncSetAttribute(k_batch_reg_smooth, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int)(SMT_WARPS * sizeof(SmoothWarp))) != cudaSuccess ||
      cudaFuncSetAttribute(k_batch_smooth_spectral, cudaFuncAttributeMaxDynamicSharedMemorySize, SMT_SPEC_SMEM) !=
          cudaSuccess)
    return BEM3_ERR_CUDA;
  bool wide = true;  // every matrix of the interior domains starts on 16 bytes
  for (int i = 0; i < n; i++)
    if (!doms[i].periodic)
      wide = wide && wide_cplx(doms[i].G) && wide_cplx(doms[i].H) && wide_cplx(doms[i].dG) && wide_cplx(doms[i].dH);
  const auto batch_reg_interior = wide ? k_batch_reg_interior<true> : k_batch_reg_interior<false>;
  if (cudaFuncSetAttribute(batch_reg_interior, cudaFuncAttributePreferredSharedMemoryCarveout,
                           (int)cudaSharedmemCarveoutMaxShared) != cudaSuccess ||
      cudaFuncSetAttribute(batch_reg_interior, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)REGI_SMEM_BYTES) !=
          cudaSuccess)
    return BEM3_ERR_CUDA;

  bem3_batch b = new bem3_batch_s;
  cudaGetDevice(&b->dev);
  b->nd = n;

  // host descriptors, lattices and propagating orders
  std::vector<BatchDomain> hD((size_t)n);
  std::vector<std::vector<QPProp>> props((size_t)n);
  SegHost selfP, selfI, regP, regI, rows, smtP;
  size_t spec_smem = 0;
  std::vector<int> pdom, idom;
  for (int i = 0; i < n; i++) {
    const bem3_batch_domain& d = doms[i];
    BatchDomain& B = hD[(size_t)i];
    memset(&B, 0, sizeof B);
    AssembleArgs& A = B.A;
    A.geo = d.geo; A.sid = d.sid; A.ne = d.Ne_d; A.did = d.did; A.periodic = d.periodic ? 1 : 0;
    A.kre = d.kre; A.kim = d.kim;
    A.G = d.G; A.H = d.H; A.dG = d.dG; A.dH = d.dH; A.dF = d.dF;
    A.terms = nullptr;
    const long long ne = d.Ne_d;
    if (A.periodic) {
      int e = lattice_from(&d.qd, &B.L);
      if (e) { batch_free(b); return e; }
      props[(size_t)i].resize(QP_PROP_CAP);
      const int np = qp_prop_list(B.L, props[(size_t)i].data(), QP_PROP_CAP);
      if (np < 0) { batch_free(b); return BEM3_ERR_LATTICE; }
      props[(size_t)i].resize((size_t)np);
      B.L.nprop = np;
      selfP.add(i, 4 * ne);
      regP.add(i, (4 * ne * ne + REGP_PAIRS - 1) / REGP_PAIRS);
      smtP.add(i, 4 * ne * ((ne + SMT_PAIRS - 1) / SMT_PAIRS));
      smooth_lattice(B.L, B.M.S);
      if (B.M.S.ok) {
        B.M.cap = batch_table_room(B.L, B.M.S, (int)ne);
        spec_smem = std::max(spec_smem, smooth_spec_smem(B.M.S));
      }
      pdom.push_back(i);
    } else {
      selfI.add(i, 4 * ne);
      regI.add(i, 4 * ne * ((ne + 31) / 32));
      idom.push_back(i);
    }
    rows.add(i, 4 * ne);
  }

  // one allocation
  Layout Lay;
  const size_t oD = Lay.take(sizeof(BatchDomain) * (size_t)n);
  const size_t oStatus = Lay.take(sizeof(int) * (size_t)n);
  const size_t oNext = Lay.take(sizeof(unsigned long long) * 4);
  constexpr int NSEG = 6;
  SegHost* segs[NSEG] = {&selfP, &selfI, &regP, &regI, &rows, &smtP};
  size_t oBase[NSEG], oDom[NSEG];
  for (int k = 0; k < NSEG; k++) {
    oBase[k] = Lay.take(sizeof(long long) * segs[k]->base.size());
    oDom[k] = Lay.take(sizeof(int) * (segs[k]->dom.size() + 1));
  }
  const size_t oPdom = Lay.take(sizeof(int) * (pdom.size() + 1));
  const size_t oIdom = Lay.take(sizeof(int) * (idom.size() + 1));
  std::vector<size_t> oFp((size_t)n), oFself((size_t)n), oList((size_t)n), oCount((size_t)n), oProp((size_t)n, 0);
  std::vector<size_t> oPool((size_t)n, 0), oIp((size_t)n, 0), oSc((size_t)n, 0);
  for (int i = 0; i < n; i++) {
    const size_t ne = (size_t)doms[i].Ne_d, np = 4 * ne * ne;
    oFp[(size_t)i] = Lay.take(np * sizeof(double3));
    oFself[(size_t)i] = Lay.take(4 * ne * sizeof(double3));
    hD[(size_t)i].gh_cap = (unsigned)(np / 8 + 4096);
    oList[(size_t)i] = Lay.take((size_t)hD[(size_t)i].gh_cap * sizeof(unsigned));
    oCount[(size_t)i] = Lay.take(sizeof(unsigned));
    if (doms[i].periodic && !props[(size_t)i].empty()) oProp[(size_t)i] = Lay.take(sizeof(QPProp) * props[(size_t)i].size());
    if (hD[(size_t)i].M.cap) {
      oIp[(size_t)i] = Lay.take(np * sizeof(unsigned));
      oSc[(size_t)i] = Lay.take(3 * sizeof(unsigned));
    }
  }
  // the pool, and the groups of periodic domains that go through it (from groups[k] to before groups[k + 1] of pdom).
  // Where the memory cannot be had: a smaller pool and more groups; domains that do not fit it, then all of them, are
  // summed point by point.
  std::vector<int> groups;
  for (size_t limit = BATCH_POOL_BYTES;; limit = limit > ((size_t)32 << 20) ? limit / 4 : 0) {
    groups.assign(1, 0);
    size_t pool = 0, at = 0;
    for (int q = 0; q < (int)pdom.size(); q++) {
      BatchDomain& B = hD[(size_t)pdom[(size_t)q]];
      if (!B.M.cap) continue;
      const size_t part = pool_part(B.M.cap, B.gh_cap).end;
      if (part > limit && limit < BATCH_POOL_BYTES) {
        B.M.cap = 0;
        continue;
      }
      if (at > 0 && at + part > limit) {
        groups.push_back(q);
        at = 0;
      }
      oPool[(size_t)pdom[(size_t)q]] = Lay.off + at;
      at += part;
      pool = std::max(pool, at);
    }
    groups.push_back((int)pdom.size());
    b->bytes = Lay.off + pool;
    if (cudaMalloc(&b->mem, b->bytes) == cudaSuccess) break;
    b->mem = nullptr;
    if (limit == 0) { batch_free(b); return BEM3_ERR_CUDA; }
    cudaGetLastError();
  }
  char* m = (char*)b->mem;
  b->dD = (BatchDomain*)(m + oD);
  b->dstatus = (int*)(m + oStatus);
  unsigned long long* next = (unsigned long long*)(m + oNext);
  for (int i = 0; i < n; i++) {
    BatchDomain& B = hD[(size_t)i];
    B.Fp = (double3*)(m + oFp[(size_t)i]);
    B.Fself = (double3*)(m + oFself[(size_t)i]);
    B.gh_list = (unsigned*)(m + oList[(size_t)i]);
    B.gh_count = (unsigned*)(m + oCount[(size_t)i]);
    B.status = b->dstatus + i;
    if (B.M.cap) {
      const PoolPart part = pool_part(B.M.cap, B.gh_cap);
      char* at = m + oPool[(size_t)i];
      B.M.plan = (SmoothPlan*)at;
      B.M.tab = (cplx*)(at + part.tab);
      B.M.smp = (cplx*)(at + part.smp);
      B.smt_list = (unsigned*)(at + part.list);
      B.ip_list = (unsigned*)(m + oIp[(size_t)i]);
      B.smt_count = (unsigned*)(m + oSc[(size_t)i]);
    }
    if (doms[i].periodic) B.L.prop = props[(size_t)i].empty() ? nullptr : (QPProp*)(m + oProp[(size_t)i]);
  }
  // uploads (synchronous: creation is outside the timed path)
  bool ok = cudaMemcpy(b->dD, hD.data(), sizeof(BatchDomain) * (size_t)n, cudaMemcpyHostToDevice) == cudaSuccess;
  BatchSeg S[NSEG];
  for (int k = 0; k < NSEG && ok; k++) {
    ok = cudaMemcpy(m + oBase[k], segs[k]->base.data(), sizeof(long long) * segs[k]->base.size(), cudaMemcpyHostToDevice) ==
         cudaSuccess;
    if (ok && !segs[k]->dom.empty())
      ok = cudaMemcpy(m + oDom[k], segs[k]->dom.data(), sizeof(int) * segs[k]->dom.size(), cudaMemcpyHostToDevice) ==
           cudaSuccess;
    S[k].base = (const long long*)(m + oBase[k]);
    S[k].dom = (const int*)(m + oDom[k]);
    S[k].n = segs[k]->n();
  }
  if (ok && !pdom.empty())
    ok = cudaMemcpy(m + oPdom, pdom.data(), sizeof(int) * pdom.size(), cudaMemcpyHostToDevice) == cudaSuccess;
  if (ok && !idom.empty())
    ok = cudaMemcpy(m + oIdom, idom.data(), sizeof(int) * idom.size(), cudaMemcpyHostToDevice) == cudaSuccess;
  for (int i = 0; i < n && ok; i++)
    if (oProp[(size_t)i])
      ok = cudaMemcpy(m + oProp[(size_t)i], props[(size_t)i].data(), sizeof(QPProp) * props[(size_t)i].size(),
                      cudaMemcpyHostToDevice) == cudaSuccess;
  if (!ok) { batch_free(b); return BEM3_ERR_CUDA; }

  // the launch sequence, captured once
  int sms = 148;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, b->dev);
  cudaStream_t s0 = nullptr, s1 = nullptr;
  cudaEvent_t fork = nullptr, join = nullptr;
  if (cudaStreamCreateWithFlags(&s0, cudaStreamNonBlocking) != cudaSuccess ||
      cudaStreamCreateWithFlags(&s1, cudaStreamNonBlocking) != cudaSuccess ||
      cudaEventCreateWithFlags(&fork, cudaEventDisableTiming) != cudaSuccess ||
      cudaEventCreateWithFlags(&join, cudaEventDisableTiming) != cudaSuccess) {
    ok = false;
  }
  int launches = 0;
  if (ok && cudaStreamBeginCapture(s0, cudaStreamCaptureModeThreadLocal) != cudaSuccess) ok = false;
  if (ok) {
    k_batch_reset<<<(n + 255) / 256, 256, 0, s0>>>(b->dD, n, next);
    k_batch_zero<<<dim3(2 * sms, (unsigned)n), 256, 0, s0>>>(b->dD);
    launches += 2;
    cudaEventRecord(fork, s0);
    cudaStreamWaitEvent(s1, fork, 0);
    // periodic branch
    for (size_t q = 0; spec_smem > 0 && q + 1 < groups.size(); q++) {
      const int p0 = groups[q], p1 = groups[q + 1];
      const unsigned npd = (unsigned)(p1 - p0);
      if (npd == 0) continue;
      const int* dp = (const int*)(m + oPdom) + p0;
      const long long r0 = selfP.base[(size_t)p0], rows = selfP.base[(size_t)p1] - r0;
      const long long u0 = smtP.base[(size_t)p0], u1 = smtP.base[(size_t)p1];
      k_batch_smooth_plan<<<npd, SMT_PLAN_THREADS, 0, s0>>>(b->dD, dp);
      k_batch_smooth_spectral<<<dim3((unsigned)(4 * sms), npd), SMT_SPEC_THREADS, spec_smem, s0>>>(b->dD, dp);
      k_batch_smooth_project<<<dim3((unsigned)(8 * sms), npd), SMT_PROJ_THREADS, 0, s0>>>(b->dD, dp);
      k_batch_self_smooth<<<(unsigned)rows, SELF_THREADS, 0, s0>>>(b->dD, S[0], r0);
      k_batch_reg_smooth<<<(unsigned)((u1 - u0 + SMT_WARPS - 1) / SMT_WARPS), SMT_WARPS * 32,
                           SMT_WARPS * sizeof(SmoothWarp), s0>>>(b->dD, S[5], u0, u1);
      k_batch_gh_smooth<<<(unsigned)(sms * T.gh_blocks_per_sm), 256, 0, s0>>>(b->dD, dp, (int)npd);
      launches += 6;
    }
    if (selfP.total() > 0) { k_batch_self_periodic<<<(unsigned)selfP.total(), SELF_THREADS, 0, s0>>>(b->dD, S[0]); launches++; }
    if (regP.total() > 0) {
      const long long want = (regP.total() * 32 + 255) / 256;  // CTAs that would give every warp one unit
      const unsigned ctas = (unsigned)std::min<long long>((long long)sms * T.regp_blocks_per_sm, std::max(want, 1LL));
      k_batch_reg_periodic<<<ctas, 256, REGP_SMEM_BYTES, s0>>>(b->dD, S[2], T.grab_units, next);
      k_batch_gh_periodic<<<(unsigned)(sms * T.gh_blocks_per_sm), 256, 0, s0>>>(b->dD, (const int*)(m + oPdom),
                                                                             (int)pdom.size());
      launches += 2;
    }
    // interior branch
    if (selfI.total() > 0) { k_batch_self_interior<<<(unsigned)selfI.total(), SI_THREADS, 0, s1>>>(b->dD, S[1]); launches++; }
    if (regI.total() > 0) {
      batch_reg_interior<<<(unsigned)((regI.total() + REGI_WARPS - 1) / REGI_WARPS), REGI_WARPS * 32, REGI_SMEM_BYTES, s1>>>(
          b->dD, S[3]);
      k_batch_gh_interior<<<(unsigned)(2 * sms * T.gh_blocks_per_sm), GHI_THREADS, 0, s1>>>(b->dD, (const int*)(m + oIdom),
                                                                             (int)idom.size());
      launches += 2;
    }
    cudaEventRecord(join, s1);
    cudaStreamWaitEvent(s0, join, 0);
    k_batch_rowsum<<<(unsigned)((rows.total() * 32 + 255) / 256), 256, 0, s0>>>(b->dD, S[4]);
    launches++;
    if (cudaGetLastError() != cudaSuccess) ok = false;
    cudaGraph_t g = nullptr;
    if (cudaStreamEndCapture(s0, &g) != cudaSuccess || !g) ok = false;
    b->graph = g;
    if (ok && cudaGraphInstantiate(&b->exec, b->graph, 0) != cudaSuccess) { b->exec = nullptr; ok = false; }
  }
  if (fork) cudaEventDestroy(fork);
  if (join) cudaEventDestroy(join);
  if (s0) cudaStreamDestroy(s0);
  if (s1) cudaStreamDestroy(s1);
  if (!ok) { batch_free(b); return BEM3_ERR_CUDA; }
  b->launches = launches;
  *out = b;
  return 0;
}

extern "C" int bem3_batch_run(bem3_batch b, void* stream)
{
  if (!b || !b->exec) return BEM3_ERR_ARG;
  return cudaGraphLaunch(b->exec, (cudaStream_t)stream) == cudaSuccess ? 0 : BEM3_ERR_CUDA;
}

extern "C" int bem3_batch_wait(bem3_batch b, void* stream, int* per_domain)
{
  if (!b) return BEM3_ERR_ARG;
  std::vector<int> st((size_t)b->nd, 0);
  cudaStream_t s = (cudaStream_t)stream;
  if (cudaMemcpyAsync(st.data(), b->dstatus, sizeof(int) * (size_t)b->nd, cudaMemcpyDeviceToHost, s) != cudaSuccess ||
      cudaStreamSynchronize(s) != cudaSuccess)
    return BEM3_ERR_CUDA;
  int first = 0;
  for (int i = 0; i < b->nd; i++) {
    if (per_domain) per_domain[i] = st[(size_t)i];
    if (!first && st[(size_t)i]) first = st[(size_t)i];
  }
  return first;
}

extern "C" int bem3_batch_info(bem3_batch b, int* launches, size_t* device_bytes)
{
  if (!b) return BEM3_ERR_ARG;
  if (launches) *launches = b->launches;
  if (device_bytes) *device_bytes = b->bytes;
  return 0;
}

extern "C" int bem3_batch_destroy(bem3_batch b)
{
  if (!b) return BEM3_ERR_ARG;
  int cur = 0;
  cudaGetDevice(&cur);
  const int dev = b->dev;
  if (cur != dev) cudaSetDevice(dev);
  batch_free(b);
  if (cur != dev) cudaSetDevice(cur);
  return 0;
}
