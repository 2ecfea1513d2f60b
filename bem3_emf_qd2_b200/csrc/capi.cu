// capi.cu -- extern "C" entry points (include/bem3_qd2_b200.h) and the per-device resources
// they share: scratch for the assembly, a status word written by the kernels.
#include <cuda_runtime.h>
#include <stdint.h>
#include <stdio.h>
#include <string.h>

#include <mutex>
#include <vector>

#include "elem.cuh"
#include "qpgf_warp.cuh"
#include "bem3_internal.h"

#define MAX_DEV 64

namespace {

struct DevRes {
  void* scratch = nullptr;
  size_t scratch_bytes = 0;
  int* status = nullptr;  // device int
  unsigned long long* terms = nullptr;  // device counter (profiling only)
  QPProp* prop = nullptr;               // propagating orders of the lattice being assembled
};

// One set per host thread and device: concurrent assemblies from different threads (each on its
// own stream) never share scratch.  A thread's scratch is kept until the thread ends.
struct ThreadRes {
  DevRes d[MAX_DEV];
  DevRes& operator[](int i) { return d[i]; }
  ~ThreadRes()
  {
    int now = -1;
    for (int i = 0; i < MAX_DEV; i++) {
      DevRes& r = d[i];
      if (!r.scratch && !r.status && !r.terms && !r.prop) continue;
      if (now < 0 && cudaGetDevice(&now) != cudaSuccess) return;  // the runtime is gone: so is the memory
      if (cudaSetDevice(i) != cudaSuccess) continue;
      cudaFree(r.scratch);
      cudaFree(r.status);
      cudaFree(r.terms);
      cudaFree(r.prop);
    }
    if (now >= 0) cudaSetDevice(now);
  }
};
thread_local ThreadRes t_res;
thread_local bem3_stats t_last_stats;
thread_local bem3_table_stats t_last_table;
thread_local int t_profiling = 0;

int cur_dev()
{
  int d = 0;
  cudaGetDevice(&d);
  return d;
}

// Grows the device scratch of the current device to at least `bytes`.
int ensure_scratch(size_t bytes, DevRes** out)
{
  int d = cur_dev();
  if (d < 0 || d >= MAX_DEV) return BEM3_ERR_ARG;
  DevRes& r = t_res[d];
  if (!r.status) {
    if (cudaMalloc(&r.status, sizeof(int)) != cudaSuccess) return BEM3_ERR_CUDA;
  }
  if (r.scratch_bytes < bytes) {
    if (r.scratch) cudaFree(r.scratch);
    r.scratch = nullptr;
    r.scratch_bytes = 0;
    if (cudaMalloc(&r.scratch, bytes) != cudaSuccess) return BEM3_ERR_CUDA;
    r.scratch_bytes = bytes;
  }
  *out = &r;
  return 0;
}

// The lattice's propagating orders into device memory `dst` (QP_PROP_CAP entries) on `st`, for
// the hoisted spectral sums of the assembly kernels.
int attach_prop_list(QPLattice* L, QPProp* dst, cudaStream_t st)
{
  static thread_local QPProp host[QP_PROP_CAP];
  const int n = qp_prop_list(*L, host, QP_PROP_CAP);
  if (n < 0) return BEM3_ERR_LATTICE;  // more propagating orders than the list holds
  L->prop = dst;
  L->nprop = n;
  if (n > 0 && cudaMemcpyAsync(dst, host, sizeof(QPProp) * (size_t)n, cudaMemcpyHostToDevice, st) != cudaSuccess)
    return BEM3_ERR_CUDA;
  return 0;
}

int lattice_from(const bem3_qpd2* qd, QPLattice* L)
{
  if (!qd) return BEM3_ERR_ARG;
  if (qp_lattice_init(*L, qd->k, qd->vk[0], qd->vk[1], qd->vd1[0], qd->vd1[1], qd->vd2[0], qd->vd2[1]) != 0)
    return BEM3_ERR_LATTICE;
  return 0;
}

}  // namespace

// ------------------------------------------------------------------------------------------
// A warp per point (qpgf_warp.cuh).  Bound by each warp's chain of batches (special functions, then sums in
// serial order), not by FP64: 24 % of the issue slots are used.  One B200, bem3_qpgf on 4,096 points (square
// lattice, 0.63 um): 2,975-3,575 -> 580 us, of which the kernel 1,900 -> 442 us; the rest is copies (the three
// allocations of each call cost 0.6 to 1.1 ms).
#define QPGF_WARPS 4
#define QPGF_CHUNK (1 << 18)
template <int MODE>
__global__ void __launch_bounds__(QPGF_WARPS * 32, 4) k_qpgf_points(const __grid_constant__ QPLattice L, int n,
                                                                 const double* __restrict__ r, double* __restrict__ out,
                                                                 int* __restrict__ ret)
{
  __shared__ QwBatch batch[QPGF_WARPS];
  const int i = blockIdx.x * QPGF_WARPS + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (i >= n) return;  // uniform across the warp
  const double p[3] = {r[3 * (size_t)i], r[3 * (size_t)i + 1], r[3 * (size_t)i + 2]};
  QPVal v;
  const int e = qpgf_eval_warp<MODE>(L, p, lane, batch[threadIdx.x >> 5], v);
  if (lane != 0) return;
  ret[i] = e;
  double* o = out + 8 * (size_t)i;
  o[0] = v.G.re; o[1] = v.G.im;
  for (int c = 0; c < 3; c++) { o[2 + 2 * c] = v.dG[c].re; o[3 + 2 * c] = v.dG[c].im; }
}

extern "C" int bem3_qpgf_dev(const bem3_qpd2* qd, int n, const double* r_dev, double* out_dev, int* ret_dev, int mode,
                             void* stream)
{
  if (n < 0 || (n > 0 && (!r_dev || !out_dev || !ret_dev))) return BEM3_ERR_ARG;
  QPLattice L;
  int e = lattice_from(qd, &L);
  if (e) return e;
  if (n == 0) return 0;
  const unsigned blocks = (unsigned)(n / QPGF_WARPS + (n % QPGF_WARPS != 0));
  if (mode == 0) k_qpgf_points<QP_V1><<<blocks, QPGF_WARPS * 32, 0, (cudaStream_t)stream>>>(L, n, r_dev, out_dev, ret_dev);
  else k_qpgf_points<QP_BOTH><<<blocks, QPGF_WARPS * 32, 0, (cudaStream_t)stream>>>(L, n, r_dev, out_dev, ret_dev);
  return cudaGetLastError() == cudaSuccess ? 0 : BEM3_ERR_CUDA;
}

extern "C" int bem3_qpgf(const bem3_qpd2* qd, int n, const double* r, double* out, int* ret, int mode)
{
  if (n < 0 || (n > 0 && (!r || !out || !ret))) return BEM3_ERR_ARG;
  if (n == 0) return 0;
  QPLattice L;
  int rc = lattice_from(qd, &L);  // before the first copy: nothing is in flight when a lattice is refused
  if (rc) return rc;
  // the points and results in this thread's scratch, QPGF_CHUNK points (24 MB) at a time
  const int chunk = n < QPGF_CHUNK ? n : QPGF_CHUNK;
  const size_t m = (size_t)chunk;
  DevRes* R = nullptr;
  if ((rc = ensure_scratch(m * (3 + 8) * sizeof(double) + m * sizeof(int), &R))) return rc;
  double* dout = (double*)R->scratch;
  double* dr = dout + 8 * m;
  int* dret = (int*)(dr + 3 * m);
  const cudaStream_t st = cudaStreamPerThread;
  for (int i = 0; rc == 0; i += chunk) {
    const int c = n - i < chunk ? n - i : chunk;
    const size_t b = (size_t)c;
    if (cudaMemcpyAsync(dr, r + 3 * (size_t)i, 3 * sizeof(double) * b, cudaMemcpyHostToDevice, st) != cudaSuccess) {
      rc = BEM3_ERR_CUDA;
    } else if ((rc = bem3_qpgf_dev(qd, c, dr, dout, dret, mode, st)) == 0 &&
               (cudaMemcpyAsync(out + 8 * (size_t)i, dout, 8 * sizeof(double) * b, cudaMemcpyDeviceToHost, st) != cudaSuccess ||
                cudaMemcpyAsync(ret + i, dret, sizeof(int) * b, cudaMemcpyDeviceToHost, st) != cudaSuccess)) {
      rc = BEM3_ERR_CUDA;
    }
    // on every way out: the copies read and write the caller's arrays
    if (cudaStreamSynchronize(st) != cudaSuccess && rc == 0) rc = BEM3_ERR_CUDA;
    if (n - i <= chunk) break;
  }
  return rc;
}

// ------------------------------------------------------------------------------------------
extern "C" int bem3_geo_stride(void) { return GEO_STRIDE; }

extern "C" int bem3_pack_geometry(const bem3_mesh* m, double* geo)
{
  if (!m || !geo || m->Ne <= 0 || !m->cr || !m->cw || !m->ren || !m->wen || !m->nv) return BEM3_ERR_ARG;
  for (int i = 0; i <= m->Ne; i++) {
    double* g = geo + (size_t)i * GEO_STRIDE;
    memset(g, 0, sizeof(double) * GEO_STRIDE);
    if (i == 0) continue;
    memcpy(g + GEO_CR, m->cr + (size_t)i * 12, 12 * sizeof(double));
    memcpy(g + GEO_CW, m->cw + (size_t)i * 9, 9 * sizeof(double));
    memcpy(g + GEO_REN, m->ren + (size_t)i * 12, 12 * sizeof(double));
    memcpy(g + GEO_WEN, m->wen + (size_t)i * 12, 12 * sizeof(double));
    int nv = m->nv[i];
    if (nv != 3 && nv != 4) return BEM3_ERR_ARG;
    g[GEO_NN] = (double)nv;
  }
  return 0;
}

extern "C" unsigned long long bem3_last_gh_pairs(void) { return t_last_stats.gh_pairs; }

extern "C" void bem3_set_profiling(int on) { t_profiling = on ? 1 : 0; }

extern "C" int bem3_last_stats(bem3_stats* out)
{
  if (!out) return BEM3_ERR_ARG;
  *out = t_last_stats;
  return 0;
}

extern "C" int bem3_last_table_stats(bem3_table_stats* out)
{
  if (!out) return BEM3_ERR_ARG;
  *out = t_last_table;
  return 0;
}

// Rows per chunk so that the per-pair scratch stays near 384 MB.
static int default_rows_per_chunk(int ne)
{
  long long rows = (16LL << 20) / (ne > 0 ? ne : 1);
  if (rows < 4) rows = 4;
  if (rows > 4LL * ne) rows = 4LL * ne;
  return (int)rows;
}

// A periodic domain's lattice and the room for its table (cap coefficients; 0: summed point by point).
struct PeriodicHost {
  QPLattice L;
  SmoothLat S;
  long long cap = 0;
};
static int periodic_host(const bem3_qpd2* qd, int ne, PeriodicHost& P)
{
  memset(&P.L, 0, sizeof P.L);
  int e = lattice_from(qd, &P.L);
  if (e) return e;
  smooth_lattice(P.L, P.S);
  P.cap = smooth_capacity(P.L, P.S, ne, 4.0 * (double)ne * ne, 144.0, 0.0);
  return 0;
}

// This thread's scratch for `rows` rows a chunk of a domain of ne elements, with `extra` bytes behind it.  The
// table is what may be left out: where the memory cannot be had, less room for it (*cap), then none.
static int table_scratch(int ne, int rows, size_t extra, long long* cap, DevRes** R)
{
  for (;;) {
    const size_t need = ((bem3_scratch_bytes(ne, rows, *cap) + 255) & ~(size_t)255) + extra;
    const int e = ensure_scratch(need, R);
    if (e != BEM3_ERR_CUDA || *cap == 0) return e;
    cudaGetLastError();  // the failed allocation's error must not be found after a later launch
    *cap = *cap > SMT_CAPMIN ? SMT_CAPMIN : 0;
  }
}

// One domain's assembly in flight on a stream: its per-thread resources and counters.
struct DomainRun {
  DevRes* R = nullptr;
  AssembleStats S;
  bool profiling = false;
};

// Enqueues the assembly of one domain on `st` (device inputs and outputs) without waiting for it;
// `hook` (optional) sees every row chunk as its kernels are enqueued.  given: the periodic domain's lattice and
// table where the caller has set them up and holds the scratch already.
static int enqueue_domain(const double* geo_dev, int Ne, const int* sid_dev, int Ne_d, int did, int periodic,
                          const bem3_qpd2* qd, double kre, double kim, double* G_dev, double* H_dev, double* dG_dev,
                          double* dH_dev, double* dF_dev, cudaStream_t st, int rows, const ChunkHook* hook,
                          DomainRun& run, const PeriodicHost* given = nullptr)
{
  if (!geo_dev || !sid_dev || Ne <= 0 || Ne_d <= 0 || Ne_d > 2 * Ne || !G_dev || !H_dev) return BEM3_ERR_ARG;
  PeriodicHost own;
  int e = 0;
  if (!periodic) given = nullptr;
  else if (!given && (e = periodic_host(qd, Ne_d, own))) return e;
  long long cap = given ? given->cap : own.cap;
  DevRes* R = nullptr;
  if ((e = table_scratch(Ne_d, rows, 0, &cap, &R))) return e;
  QPLattice L = given ? given->L : own.L;
  const SmoothLat* S = given ? &given->S : periodic ? &own.S : nullptr;
  AssembleArgs A;
  A.geo = geo_dev; A.sid = sid_dev; A.ne = Ne_d; A.did = did; A.periodic = periodic ? 1 : 0;
  A.kre = kre; A.kim = kim;
  A.G = G_dev; A.H = H_dev; A.dG = dG_dev; A.dH = dH_dev; A.dF = dF_dev;
  if (periodic) {
    if (!R->prop && cudaMalloc(&R->prop, sizeof(QPProp) * QP_PROP_CAP) != cudaSuccess) return BEM3_ERR_CUDA;
    if ((e = attach_prop_list(&L, R->prop, st))) return e;
  }
  if (cudaMemsetAsync(R->status, 0, sizeof(int), st) != cudaSuccess) return BEM3_ERR_CUDA;
  A.terms = nullptr;
  run.profiling = t_profiling != 0;
  if (run.profiling) {
    if (!R->terms && cudaMalloc(&R->terms, sizeof(unsigned long long)) != cudaSuccess) return BEM3_ERR_CUDA;
    A.terms = R->terms;
    cudaMemsetAsync(R->terms, 0, sizeof(unsigned long long), st);
  }
  memset(&run.S, 0, sizeof run.S);
  run.S.time_kernels = t_profiling;
  run.R = R;
  return bem3_assemble_run(A, &L, S, R->scratch, R->scratch_bytes, rows, cap, R->status, st, &run.S, hook);
}

// Waits for `st` and returns the kernels' status; fills this thread's counters.
static int finish_domain(cudaStream_t st, const DomainRun& run)
{
  int hs = 0;
  unsigned long long terms = 0, gh = 0;
  if (cudaMemcpyAsync(&hs, run.R->status, sizeof(int), cudaMemcpyDeviceToHost, st) != cudaSuccess) return BEM3_ERR_CUDA;
  if (run.profiling && cudaMemcpyAsync(&terms, run.R->terms, sizeof terms, cudaMemcpyDeviceToHost, st) != cudaSuccess)
    return BEM3_ERR_CUDA;
  if (cudaMemcpyAsync(&gh, run.S.d_gh_total, sizeof gh, cudaMemcpyDeviceToHost, st) != cudaSuccess) return BEM3_ERR_CUDA;
  if (cudaStreamSynchronize(st) != cudaSuccess) return BEM3_ERR_CUDA;
  memset(&t_last_stats, 0, sizeof t_last_stats);
  memset(&t_last_table, 0, sizeof t_last_table);
  t_last_stats.gh_pairs = gh;
  t_last_stats.qpgf_terms = terms;
  t_last_stats.launches = run.S.launches;
  t_last_stats.reg_periodic_launches = run.S.reg_periodic_launches;
  t_last_stats.reg_periodic_ms = run.S.reg_periodic_ms;
  for (int i = 0; i < 4; i++) t_last_stats.class_ms[i] = run.S.class_ms[i];
  t_last_table.on = run.S.table_on;
  t_last_table.plane_pairs = run.S.plane_pairs;
  t_last_table.reg_smooth_ms = run.S.reg_smooth_ms;
  return hs;
}

extern "C" int bem3_assemble_domain_dev(const double* geo_dev, int Ne, const int* sid_dev, int Ne_d, int did, int periodic,
                                        const bem3_qpd2* qd, double kre, double kim, double* G_dev, double* H_dev,
                                        double* dG_dev, double* dH_dev, double* dF_dev, void* stream)
{
  cudaStream_t st = (cudaStream_t)stream;
  DomainRun run;
  int e = enqueue_domain(geo_dev, Ne, sid_dev, Ne_d, did, periodic, qd, kre, kim, G_dev, H_dev, dG_dev, dH_dev, dF_dev,
                         st, default_rows_per_chunk(Ne_d), nullptr, run);
  if (e) return e;
  return finish_domain(st, run);
}

namespace {
// Row chunks finished on the device, copied to the caller's host matrices on a copy stream as soon
// as each chunk's kernels have run: the transfer of chunk c overlaps the computation of the chunks
// after it.  (To page-locked host memory the copies are asynchronous; to pageable memory each copy
// call returns once done, while the GPU keeps computing the chunks already enqueued.)
struct RowCopies {
  size_t N = 0;
  std::vector<cudaEvent_t> ev;
  std::vector<int> r0, nr;
  bool failed = false;
  static void hook(void* user, int r0, int nr, cudaStream_t st)
  {
    RowCopies& c = *(RowCopies*)user;
    cudaEvent_t e = nullptr;
    if (cudaEventCreateWithFlags(&e, cudaEventDisableTiming) != cudaSuccess || cudaEventRecord(e, st) != cudaSuccess) {
      c.failed = true;
      if (e) cudaEventDestroy(e);
      return;
    }
    c.ev.push_back(e);
    c.r0.push_back(r0);
    c.nr.push_back(nr);
  }
  ~RowCopies()
  {
    for (cudaEvent_t e : ev) cudaEventDestroy(e);
  }
};
}  // namespace

// Rows per chunk where finished chunks are copied to the host during the later ones: about 8 chunks a
// domain, fewer (down to 4) where a chunk would not give the GPU two rounds of the regular kernel's warps
// (16 a multiprocessor with 4 sources each, 9 with 32).  At least 64 rows.
static int copied_rows_per_chunk(int Ne, bool periodic)
{
  const int N = 4 * Ne, wpr = periodic ? (Ne + 3) / 4 : (Ne + 31) / 32;
  const int fill = (2 * 148 * (periodic ? 16 : 9) + wpr - 1) / wpr;
  int r = (N + 7) / 8;
  const int most = (N + 3) / 4;
  if (r < fill) r = fill < most ? fill : most;
  if (r < 64) r = 64;
  const int top = default_rows_per_chunk(Ne);
  return r > top ? top : r;
}

extern "C" int bem3_assemble_domain(const bem3_mesh* mesh, const int* sid, int Ne_d, int did, int periodic,
                                    const bem3_qpd2* qd, double kre, double kim, double* G, double* H, double* dG,
                                    double* dH, double* dF)
{
  if (!mesh || !sid || Ne_d <= 0 || !G || !H) return BEM3_ERR_ARG;
  for (int i = 0; i < Ne_d; i++)
    if (sid[i] == 0 || sid[i] > mesh->Ne || -sid[i] > mesh->Ne) return BEM3_ERR_ARG;
  const int Ne = mesh->Ne;
  std::vector<double> geo((size_t)(Ne + 1) * GEO_STRIDE);
  int e = bem3_pack_geometry(mesh, geo.data());
  if (e) return e;
  const size_t N = (size_t)4 * Ne_d;
  double *dgeo = nullptr, *dG_ = nullptr, *dH_ = nullptr, *ddG = nullptr, *ddH = nullptr, *ddF = nullptr;
  int* dsid = nullptr;
  cudaStream_t cs = nullptr;
  int rc = BEM3_ERR_CUDA;
  RowCopies rcp;
  rcp.N = N;
  const ChunkHook hook = {RowCopies::hook, &rcp};
  const int rows = copied_rows_per_chunk(Ne_d, periodic != 0);
  DomainRun run;
  if (cudaStreamCreateWithFlags(&cs, cudaStreamNonBlocking) != cudaSuccess) { cs = nullptr; goto done; }
  if (cudaMalloc(&dgeo, geo.size() * sizeof(double)) != cudaSuccess) goto done;
  if (cudaMalloc(&dsid, Ne_d * sizeof(int)) != cudaSuccess) goto done;
  if (cudaMalloc(&dG_, N * N * 16) != cudaSuccess) goto done;
  if (cudaMalloc(&dH_, N * N * 16) != cudaSuccess) goto done;
  if (dG && cudaMalloc(&ddG, 2 * N * N * 16) != cudaSuccess) goto done;
  if (dH && cudaMalloc(&ddH, 2 * N * N * 16) != cudaSuccess) goto done;
  if (dF && cudaMalloc(&ddF, 3 * N * sizeof(double)) != cudaSuccess) goto done;
  if (cudaMemcpy(dgeo, geo.data(), geo.size() * sizeof(double), cudaMemcpyHostToDevice) != cudaSuccess) goto done;
  if (cudaMemcpy(dsid, sid, Ne_d * sizeof(int), cudaMemcpyHostToDevice) != cudaSuccess) goto done;
  rc = enqueue_domain(dgeo, Ne, dsid, Ne_d, did, periodic, qd, kre, kim, dG_, dH_, ddG, ddH, ddF, nullptr, rows, &hook,
                      run);
  if (rc) goto done;
  rc = BEM3_ERR_CUDA;
  if (rcp.failed) goto done;
  for (size_t c = 0; c < rcp.ev.size(); c++) {
    const size_t a = (size_t)rcp.r0[c], n = (size_t)rcp.nr[c];
    if (cudaStreamWaitEvent(cs, rcp.ev[c], 0) != cudaSuccess) goto done;
    if (cudaMemcpyAsync(G + 2 * a * N, dG_ + 2 * a * N, n * N * 16, cudaMemcpyDeviceToHost, cs) != cudaSuccess) goto done;
    if (cudaMemcpyAsync(H + 2 * a * N, dH_ + 2 * a * N, n * N * 16, cudaMemcpyDeviceToHost, cs) != cudaSuccess) goto done;
    if (dG && cudaMemcpyAsync(dG + 4 * a * N, ddG + 4 * a * N, 2 * n * N * 16, cudaMemcpyDeviceToHost, cs) != cudaSuccess)
      goto done;
    if (dH && cudaMemcpyAsync(dH + 4 * a * N, ddH + 4 * a * N, 2 * n * N * 16, cudaMemcpyDeviceToHost, cs) != cudaSuccess)
      goto done;
    if (dF && cudaMemcpyAsync(dF + 3 * a, ddF + 3 * a, 3 * n * sizeof(double), cudaMemcpyDeviceToHost, cs) != cudaSuccess)
      goto done;
  }
  if (cudaStreamSynchronize(cs) != cudaSuccess) goto done;
  rc = finish_domain(nullptr, run);
done:
  if (cs) { cudaStreamSynchronize(cs); cudaStreamDestroy(cs); }
  cudaDeviceSynchronize();  // nothing of this call may still use the buffers freed below
  cudaFree(dgeo); cudaFree(dsid); cudaFree(dG_); cudaFree(dH_); cudaFree(ddG); cudaFree(ddH); cudaFree(ddF);
  return rc;
}

// Matrices and inputs of bem3_assemble_domains up to this size stay in the thread's scratch between calls.
#define DOMAINS_KEPT_BYTES ((size_t)512 << 20)

// Every domain of a problem through host pointers: the reference's create_cmatrix, the loop of
// create_cmatrix_domain over did = 0..MN (d3qd2_solve_bieq.c:155-163).  The domains' kernels run back
// to back on this thread's stream, the interior domains first: their matrices are large and quick to
// compute, and the open region's long lattice sums then hide their copies.  Every finished row chunk
// of every domain is copied on one copy stream while the later chunks compute, so only the open
// region's last chunk is copied after the kernels end.  All domains' device matrices are held at once.
extern "C" int bem3_assemble_domains(const bem3_mesh* mesh, int MN, const int* const* sid, const int* Ne_d, int periodic,
                                     const bem3_qpd2* qd, const double* kn, double* const* G, double* const* H,
                                     double* const* dG, double* const* dH, double* const* dF)
{
  if (!mesh || MN < 0 || !sid || !Ne_d || !kn || !G || !H) return BEM3_ERR_ARG;
  const int Ne = mesh->Ne, nd = MN + 1;
  for (int d = 0; d < nd; d++) {
    if (!sid[d] || Ne_d[d] <= 0 || !G[d] || !H[d]) return BEM3_ERR_ARG;
    for (int i = 0; i < Ne_d[d]; i++)
      if (sid[d][i] == 0 || sid[d][i] > Ne || -sid[d][i] > Ne) return BEM3_ERR_ARG;
  }
  auto opt = [](double* const* a, int d) { return a ? a[d] : nullptr; };
  std::vector<double> geo((size_t)(Ne + 1) * GEO_STRIDE);
  int e = bem3_pack_geometry(mesh, geo.data());
  if (e) return e;
  std::vector<int> order;  // interior domains first, the open region (did 0) last
  for (int d = 1; d < nd; d++) order.push_back(d);
  order.push_back(0);
  std::vector<size_t> N(nd);
  std::vector<int> rows(nd);
  PeriodicHost per;
  if (periodic && (e = periodic_host(qd, Ne_d[0], per))) return e;
  size_t need = 0;  // of the domains without a table
  for (int d = 0; d < nd; d++) {
    N[d] = (size_t)4 * Ne_d[d];
    rows[d] = copied_rows_per_chunk(Ne_d[d], periodic && d == 0);
    const size_t b = bem3_scratch_bytes(Ne_d[d], rows[d], 0);
    need = b > need ? b : need;
  }
  double* dgeo = nullptr;
  int* dstat = nullptr;
  unsigned long long* dgh = nullptr;
  std::vector<int*> dsid(nd, nullptr);
  std::vector<double*> dG_(nd, nullptr), dH_(nd, nullptr), ddG(nd, nullptr), ddH(nd, nullptr), ddF(nd, nullptr);
  std::vector<RowCopies> rcp(nd);
  std::vector<DomainRun> run(nd);
  std::vector<int> hs(nd, 0);
  std::vector<unsigned long long> hgh(nd, 0);
  cudaStream_t cs = nullptr;
  const cudaStream_t st = cudaStreamPerThread;
  int rc = BEM3_ERR_CUDA;
  DevRes* R = nullptr;
  void* own = nullptr;
  // the matrices and inputs in one piece: behind the scratch where they are small (13 allocations and
  // their release take 5.3 ms, the whole call for 216 quads 7.5 ms without them), else allocated here
  size_t bytes = 0;
  auto take = [&](size_t b) {
    const size_t at = bytes;
    bytes += (b + 255) & ~(size_t)255;
    return at;
  };
  const size_t ogeo = take(geo.size() * sizeof(double)), ostat = take(nd * sizeof(int)), ogh = take(nd * sizeof(unsigned long long));
  std::vector<size_t> osid(nd), oG(nd), oH(nd), odG(nd), odH(nd), odF(nd);
  for (int d = 0; d < nd; d++) {
    const size_t n2 = N[d] * N[d] * 16;
    osid[d] = take(Ne_d[d] * sizeof(int));
    oG[d] = take(n2);
    oH[d] = take(n2);
    if (opt(dG, d)) odG[d] = take(2 * n2);
    if (opt(dH, d)) odH[d] = take(2 * n2);
    if (opt(dF, d)) odF[d] = take(3 * N[d] * sizeof(double));
  }
  const bool kept = bytes <= DOMAINS_KEPT_BYTES;
  char* base = nullptr;
  need = (need + 255) & ~(size_t)255;
  // the scratch at its largest before the first launch: no domain may reallocate it under another's kernels
  {
    const size_t first = (bem3_scratch_bytes(Ne_d[0], rows[0], per.cap) + 255) & ~(size_t)255;
    const size_t more = need > first ? need - first : 0;  // another domain's scratch where it is the larger
    if ((rc = table_scratch(Ne_d[0], rows[0], more + (kept ? bytes : 0), &per.cap, &R))) goto done;
    const size_t now = (bem3_scratch_bytes(Ne_d[0], rows[0], per.cap) + 255) & ~(size_t)255;
    need = now > need ? now : need;
    if ((rc = ensure_scratch(need + (kept ? bytes : 0), &R))) goto done;  // with a smaller table another may need more
  }
  rc = BEM3_ERR_CUDA;
  if (!kept && cudaMalloc(&own, bytes) != cudaSuccess) { own = nullptr; goto done; }
  base = kept ? (char*)R->scratch + need : (char*)own;
  if (cudaStreamCreateWithFlags(&cs, cudaStreamNonBlocking) != cudaSuccess) { cs = nullptr; goto done; }
  dgeo = (double*)(base + ogeo);
  dstat = (int*)(base + ostat);
  dgh = (unsigned long long*)(base + ogh);
  for (int d = 0; d < nd; d++) {
    dsid[d] = (int*)(base + osid[d]);
    dG_[d] = (double*)(base + oG[d]);
    dH_[d] = (double*)(base + oH[d]);
    if (opt(dG, d)) ddG[d] = (double*)(base + odG[d]);
    if (opt(dH, d)) ddH[d] = (double*)(base + odH[d]);
    if (opt(dF, d)) ddF[d] = (double*)(base + odF[d]);
    if (cudaMemcpy(dsid[d], sid[d], Ne_d[d] * sizeof(int), cudaMemcpyHostToDevice) != cudaSuccess) goto done;
    rcp[d].N = N[d];
  }
  if (cudaMemcpy(dgeo, geo.data(), geo.size() * sizeof(double), cudaMemcpyHostToDevice) != cudaSuccess) goto done;
  for (int d : order) {
    const ChunkHook hook = {RowCopies::hook, &rcp[d]};
    rc = enqueue_domain(dgeo, Ne, dsid[d], Ne_d[d], d, (periodic && d == 0) ? 1 : 0, qd, kn[2 * d], kn[2 * d + 1],
                        dG_[d], dH_[d], ddG[d], ddH[d], ddF[d], st, rows[d], &hook, run[d], periodic && d == 0 ? &per : nullptr);
    if (rc) goto done;
    rc = BEM3_ERR_CUDA;
    if (rcp[d].failed) goto done;
    // the domain's status word and near-singular count, kept before the next domain resets them
    if (cudaMemcpyAsync(dstat + d, run[d].R->status, sizeof(int), cudaMemcpyDeviceToDevice, st) != cudaSuccess ||
        cudaMemcpyAsync(dgh + d, run[d].S.d_gh_total, sizeof(unsigned long long), cudaMemcpyDeviceToDevice, st) !=
            cudaSuccess)
      goto done;
    const size_t n = N[d];
    for (size_t c = 0; c < rcp[d].ev.size(); c++) {
      const size_t a = (size_t)rcp[d].r0[c], m = (size_t)rcp[d].nr[c];
      if (cudaStreamWaitEvent(cs, rcp[d].ev[c], 0) != cudaSuccess) goto done;
      if (cudaMemcpyAsync(G[d] + 2 * a * n, dG_[d] + 2 * a * n, m * n * 16, cudaMemcpyDeviceToHost, cs) != cudaSuccess)
        goto done;
      if (cudaMemcpyAsync(H[d] + 2 * a * n, dH_[d] + 2 * a * n, m * n * 16, cudaMemcpyDeviceToHost, cs) != cudaSuccess)
        goto done;
      if (ddG[d] &&
          cudaMemcpyAsync(dG[d] + 4 * a * n, ddG[d] + 4 * a * n, 2 * m * n * 16, cudaMemcpyDeviceToHost, cs) != cudaSuccess)
        goto done;
      if (ddH[d] &&
          cudaMemcpyAsync(dH[d] + 4 * a * n, ddH[d] + 4 * a * n, 2 * m * n * 16, cudaMemcpyDeviceToHost, cs) != cudaSuccess)
        goto done;
      if (ddF[d] &&
          cudaMemcpyAsync(dF[d] + 3 * a, ddF[d] + 3 * a, 3 * m * sizeof(double), cudaMemcpyDeviceToHost, cs) != cudaSuccess)
        goto done;
    }
  }
  if (cudaStreamSynchronize(cs) != cudaSuccess || cudaStreamSynchronize(st) != cudaSuccess) goto done;
  if (cudaMemcpy(hs.data(), dstat, nd * sizeof(int), cudaMemcpyDeviceToHost) != cudaSuccess ||
      cudaMemcpy(hgh.data(), dgh, nd * sizeof(unsigned long long), cudaMemcpyDeviceToHost) != cudaSuccess)
    goto done;
  memset(&t_last_stats, 0, sizeof t_last_stats);
  memset(&t_last_table, 0, sizeof t_last_table);
  for (int d = 0; d < nd; d++) {
    t_last_stats.gh_pairs += hgh[d];
    t_last_stats.launches += run[d].S.launches;
    t_last_stats.reg_periodic_launches += run[d].S.reg_periodic_launches;
  }
  rc = 0;
  for (int d = 0; d < nd; d++)
    if (hs[d]) { rc = hs[d]; break; }
done:
  if (cs) { cudaStreamSynchronize(cs); cudaStreamDestroy(cs); }
  cudaStreamSynchronize(st);  // nothing of this call may still use its buffers
  cudaFree(own);
  return rc;
}

// ------------------------------------------------------------------------------------------
// FP64 peak probe: independent DFMA chains, 8 per thread, sized so the launch runs ~100 ms.
__global__ void __launch_bounds__(256) k_dfma_probe(double* out, int iters, double a, double b)
{
  double x0 = threadIdx.x * 1e-9, x1 = x0 + 1e-9, x2 = x0 + 2e-9, x3 = x0 + 3e-9;
  double x4 = x0 + 4e-9, x5 = x0 + 5e-9, x6 = x0 + 6e-9, x7 = x0 + 7e-9;
  for (int i = 0; i < iters; i++) {
#pragma unroll
    for (int u = 0; u < 16; u++) {
      x0 = fma(x0, a, b); x1 = fma(x1, a, b); x2 = fma(x2, a, b); x3 = fma(x3, a, b);
      x4 = fma(x4, a, b); x5 = fma(x5, a, b); x6 = fma(x6, a, b); x7 = fma(x7, a, b);
    }
  }
  double s = x0 + x1 + x2 + x3 + x4 + x5 + x6 + x7;
  if (s == 12345.6789) out[blockIdx.x] = s;  // keeps the chains live; never true in practice
}

extern "C" double bem3_fp64_peak_tflops(void)
{
  int dev = cur_dev(), sms = 0;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  double* d = nullptr;
  if (cudaMalloc(&d, sizeof(double) * sms * 8) != cudaSuccess) return -1.0;
  const int blocks = sms * 8, iters = 4096;
  k_dfma_probe<<<blocks, 256>>>(d, 16, 0.999999, 1e-7);  // warm-up
  cudaEvent_t e0, e1;
  cudaEventCreate(&e0);
  cudaEventCreate(&e1);
  cudaEventRecord(e0);
  k_dfma_probe<<<blocks, 256>>>(d, iters, 0.999999, 1e-7);
  cudaEventRecord(e1);
  cudaEventSynchronize(e1);
  float ms = 0.f;
  cudaEventElapsedTime(&ms, e0, e1);
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  cudaFree(d);
  double flops = 2.0 * 8 * 16 * (double)iters * blocks * 256;
  return ms > 0 ? flops / (ms * 1e-3) / 1e12 : -1.0;
}

extern "C" const char* bem3_version(void) { return "bem3_emf_qd2_b200 0.1 (sm_100a, FP64)"; }

// ------------------------------------------------------------------------------------------
// Assembly without device allocation.
//
// Some callers cannot call cudaMalloc: a serving process that hands every byte of HBM out of
// its own pool under a fixed budget (allocations outside the pool are forbidden), or a
// pipeline that must not hit the implicit device-wide synchronisation cudaMalloc/cudaFree can
// cause.  For them the per-call scratch of the assembly (the chunk's F row-sum terms, the
// near-singular work list, the status word) lives in this file-scope device array instead of
// the cudaMalloc'd pool used by bem3_assemble_domain_dev.  Every GPU that loads the library
// holds the array (BEM3_NOALLOC_SCRATCH_BYTES) until the process exits.
#define BEM3_NOALLOC_SCRATCH_BYTES (32u << 20)
static __device__ __align__(256) unsigned char g_noalloc_scratch[BEM3_NOALLOC_SCRATCH_BYTES];
static void* g_noalloc_addr[MAX_DEV];  // device address of g_noalloc_scratch, per device
static std::mutex g_noalloc_mu;

extern "C" int bem3_assemble_domain_dev_noalloc(const double* geo_dev, int Ne, const int* sid_dev, int Ne_d, int did,
                                                int periodic, const bem3_qpd2* qd, double kre, double kim,
                                                double* G_dev, double* H_dev, double* dG_dev, double* dH_dev,
                                                double* dF_dev, void* stream)
{
  if (!geo_dev || !sid_dev || Ne <= 0 || Ne_d <= 0 || Ne_d > 2 * Ne || !G_dev || !H_dev) return BEM3_ERR_ARG;
  QPLattice L;
  SmoothLat S;
  memset(&L, 0, sizeof L);
  if (periodic) {
    int e = lattice_from(qd, &L);
    if (e) return e;
    smooth_lattice(L, S);
  }
  // The array's device address: host code may not use the symbol itself (that is a host-side
  // stand-in, not a device pointer), so resolve it once per device with that device current.
  const int dev = cur_dev();
  if (dev < 0 || dev >= MAX_DEV) return BEM3_ERR_ARG;
  void* base = nullptr;
  {
    std::lock_guard<std::mutex> lk(g_noalloc_mu);
    if (!g_noalloc_addr[dev]) {
      void* p = nullptr;
      if (cudaGetSymbolAddress(&p, g_noalloc_scratch) != cudaSuccess || !p) return BEM3_ERR_CUDA;
      g_noalloc_addr[dev] = p;
    }
    base = g_noalloc_addr[dev];
  }
  // [0, 256): status word; then the lattice's propagating orders; then the assembly scratch,
  // chunked to fit
  int* status = (int*)base;
  QPProp* prop = (QPProp*)((char*)base + 256);
  const size_t head = 256 + sizeof(QPProp) * QP_PROP_CAP;
  void* scratch = (char*)base + head;
  const size_t avail = BEM3_NOALLOC_SCRATCH_BYTES - head;
  int rows = default_rows_per_chunk(Ne_d);
  while (rows > 4 && bem3_scratch_bytes(Ne_d, rows, 0) > avail) rows = rows / 2 > 4 ? rows / 2 : 4;
  if (bem3_scratch_bytes(Ne_d, rows, 0) > avail) return BEM3_ERR_SCRATCH;  // domain too large for the array
  // a table of up to SMT_CAPMIN coefficients where at least 64 rows still fit beside it
  long long cap = 0;
  if (periodic) {
    int rc = default_rows_per_chunk(Ne_d);
    while (rc > 64 && bem3_scratch_bytes(Ne_d, rc, SMT_CAPMIN) > avail) rc = rc / 2 > 64 ? rc / 2 : 64;
    if (bem3_scratch_bytes(Ne_d, rc, SMT_CAPMIN) <= avail) { cap = SMT_CAPMIN; rows = rc; }
  }
  cudaStream_t st = (cudaStream_t)stream;
  AssembleArgs A;
  A.geo = geo_dev; A.sid = sid_dev; A.ne = Ne_d; A.did = did; A.periodic = periodic ? 1 : 0;
  A.kre = kre; A.kim = kim;
  A.G = G_dev; A.H = H_dev; A.dG = dG_dev; A.dH = dH_dev; A.dF = dF_dev;
  A.terms = nullptr;
  if (periodic) {
    int e2 = attach_prop_list(&L, prop, st);
    if (e2) return e2;
  }
  // the array keeps the previous call's contents: the status word must start at zero (the
  // run itself clears its row-sum slots and work-list counter before use)
  if (cudaMemsetAsync(status, 0, sizeof(int), st) != cudaSuccess) return BEM3_ERR_CUDA;
  AssembleStats run;
  memset(&run, 0, sizeof run);
  int e = bem3_assemble_run(A, &L, periodic ? &S : nullptr, scratch, avail, rows, cap, status, st, &run);
  if (e) return e;
  int hs = 0;
  unsigned long long gh = 0;
  if (cudaMemcpyAsync(&hs, status, sizeof(int), cudaMemcpyDeviceToHost, st) != cudaSuccess) return BEM3_ERR_CUDA;
  if (cudaMemcpyAsync(&gh, run.d_gh_total, sizeof gh, cudaMemcpyDeviceToHost, st) != cudaSuccess) return BEM3_ERR_CUDA;
  if (cudaStreamSynchronize(st) != cudaSuccess) return BEM3_ERR_CUDA;
  // this thread's counters, as the allocating entry fills them (no term counter or kernel timing:
  // bem3_set_profiling does not apply to this entry point)
  memset(&t_last_stats, 0, sizeof t_last_stats);
  memset(&t_last_table, 0, sizeof t_last_table);
  t_last_stats.gh_pairs = gh;
  t_last_stats.launches = run.launches;
  return hs;
}
