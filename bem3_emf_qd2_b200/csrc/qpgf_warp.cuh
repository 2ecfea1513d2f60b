// qpgf_warp.cuh -- d3hm_qpgf_d2_v1 / (qG, dqG) at a point by a whole warp, with the reference's term
// order, stop rules and term counts (qpgf.cuh; device only).
//
// The reference sums a row of the lattice from its centre outwards, one side after the other, and ends a
// side at the first term that is negligible against the sum so far.  One thread a point is a serial
// chain of 60 to 600 terms (1.9 ms for 4,096 points, whose 128 warps leave most of the GPU idle).  Here the
// lanes evaluate a row's next 32 terms at once; the sums themselves are then taken term by term, in the
// reference's order, a component to a lane, and the stop rule is applied to all of them at once: the first
// lane whose term stops ends the side.
// The row rule decides on the last bits of the sums, so they must round as the serial ones do: the terms'
// phases are multiplied up along the row exactly as there, and nothing is added in another order.
// Terms past the stop are dropped.  At z within SMT_ZPLANE periods of 0 every lane runs the serial sums
// (their rules compare rounding noise, and rows are short).
#pragma once

#include "smooth.cuh"

// One term: F, dF[3]; e: 1 evanescent or real-space (stop rule applies), 0 propagating, < 0 an error.
struct QwTerm {
  cplx F, dF[3];
  int e;
};

struct QwSum {
  double v[8];  // S, dS[0..2] (re, im)
  __device__ __forceinline__ cplx S() const { return mk(v[0], v[1]); }
  __device__ __forceinline__ cplx d(int i) const { return mk(v[2 + 2 * i], v[3 + 2 * i]); }
};

// The warp's terms of a batch, component (F, dF[0..2] as re, im) by lane, then the sums up to each.
struct QwBatch {
  double v[32][9];  // padded: a component is read by one lane, written by another
};

// Stop rule of a term against the sums s (components as QwBatch).  KIND 0: real-space sum; 1: Ewald spectral
// sum; 2: Fourier-domain sum.
template <int MODE, int KIND>
__device__ __forceinline__ bool qw_stop(const QwTerm& t, const double* s, double eps)
{
  const cplx S = mk(s[0], s[1]), d0 = mk(s[2], s[3]), d1 = mk(s[4], s[5]), d2 = mk(s[6], s[7]);
  bool stop;
  if (KIND == 0) {
    stop = qp_diff(t.F, S, eps);
    if (MODE == QP_BOTH) stop = stop && qp_diff(t.dF[0], d0, eps) && qp_diff(t.dF[1], d1, eps);
  } else {
    stop = qp_diff(t.dF[2], d2, eps);
    if (MODE == QP_BOTH) stop = stop && qp_diff(t.F, S, eps);
  }
  return t.e == 1 && stop;
}

// Term at row n, position m of the sums, phase ce: see qp_ew1_term, qp_ew2_term, qp_fd_term.
template <int KIND>
__device__ __forceinline__ void qw_term(const QPLattice& L, const double* r, double veps, int n, int m, cplx ce,
                                        QwTerm& t)
{
  if (KIND == 0) {
    qp_ew1_term(L, r, veps, n, m, ce, t.F, t.dF);
    t.e = 1;
  } else {
    t.e = (KIND == 2) ? qp_fd_term(L, r, n, m, ce, t.F, t.dF) : qp_ew2_term(L, r, veps, n, m, ce, t.F, t.dF);
  }
}

// The sum S over the lattice; returns the number of terms or the reference's error code of the sum.
template <int MODE, int KIND>
__device__ __noinline__ int qw_sum(const QPLattice& L, const double* r_in, double veps, double eps, int lane, QwBatch& B,
                                   QwSum& out)
{
  const double r[3] = {r_in[0], r_in[1], r_in[2]};
  constexpr int LIMIT = (KIND == 2) ? QP_FD_LIMIT : QP_EW_LIMIT;
  constexpr int ELIM = (KIND == 1) ? -2 : -1;
  if (KIND == 2 && r[2] == 0.0) return -4;
  QwSum S;
  for (int i = 0; i < 8; i++) S.v[i] = 0.0;
  double mine = 0.0;  // component `lane` of S (lanes 0 .. 7)
  // phase step along a row
  const cplx step = (KIND == 0) ? L.eb2 : expi(L.g2x * r[0] + L.g2y * r[1]);
  const int nc = (KIND == 0) ? 0 : L.nc1;
  int cc = 0, dir = 0, n = nc;
  for (;;) {
    QwSum old = S;
    int c;
    if (KIND == 0)
      c = -(int)round(((r[0] + (double)n * L.d1x) * L.d2x + (r[1] + (double)n * L.d1y) * L.d2y) / L.ad22);
    else if (KIND == 2)
      c = (int)round((L.vkx * L.g2x + L.vky * L.g2y - (double)n * L.g12) / L.g22);
    else
      c = (int)round(-((-L.vkx + (double)n * L.g1x) * L.g2x + (-L.vky + (double)n * L.g1y) * L.g2y) / L.g22);
    cplx ce0;
    if (KIND == 0)
      ce0 = expi(L.vkx * ((double)n * L.d1x + (double)c * L.d2x) + L.vky * ((double)n * L.d1y + (double)c * L.d2y));
    else
      ce0 = expi((-L.vkx + (double)n * L.g1x + (double)c * L.g2x) * r[0] + (-L.vky + (double)n * L.g1y + (double)c * L.g2y) * r[1]);
    int flg = 0;
    cplx ce;   // the lane's phase
    QwTerm t;  // and term
    // evaluates the lane's term at offset o (signed), whose phase is `from` times the step (its conjugate
    // for o < 0) `times` times
    auto eval = [&](int o, cplx from, int times) {
      const cplx st = o < 0 ? conj(step) : step;
      ce = from;
      for (int i = 0; i < times; i++) ce = ce * st;
      qw_term<KIND>(L, r, veps, n, c + o, ce, t);
      __syncwarp();
      B.v[lane][0] = t.F.re; B.v[lane][1] = t.F.im;
#pragma unroll
      for (int i = 0; i < 3; i++) { B.v[lane][2 + 2 * i] = t.dF[i].re; B.v[lane][3 + 2 * i] = t.dF[i].im; }
    };
    // adds the terms lo .. hi, whose offsets (unsigned) start at off0, up to the first that ends the side:
    // 1 ended, 0 not yet, < 0 error
    auto take = [&](int lo, int hi, int off0) -> int {
      __syncwarp();
      if (lane < 8) {
        double a = mine;
        for (int j = lo; j <= hi; j++) {
          a += B.v[j][lane];
          B.v[j][lane] = a;
        }
      }
      __syncwarp();
      const bool in = lane >= lo && lane <= hi;
      const int off = off0 + lane - lo;
      const bool bad = in && t.e < 0;
      const bool stop = in && off > 0 && t.e >= 0 && qw_stop<MODE, KIND>(t, B.v[lane], eps);
      const bool lim = in && off > 0 && !stop && off + 1 >= LIMIT;  // the reference gives up here
      const unsigned mb = __ballot_sync(0xffffffffu, bad), ms = __ballot_sync(0xffffffffu, stop),
                     ml = __ballot_sync(0xffffffffu, lim), mp = __ballot_sync(0xffffffffu, in && off > 0 && t.e == 0);
      const unsigned any = mb | ms | ml;
      const int end = any ? __ffs(any) - 1 : hi;
      if (mb >> end & 1) return __shfl_sync(0xffffffffu, t.e, end);
      if (any && !(ms >> end & 1)) return ELIM;
      cc += end - lo + 1;
      flg += __popc(mp & (0xffffffffu >> (31 - end)));
      if (lane < 8) mine = B.v[end][lane];
      return any ? 1 : 0;
    };
    // lanes 0 .. W: the centre and offsets 1 .. W of the first side; W + 1 .. 2 W: 1 .. W of the second.  The
    // real-space sum's sides end after 3 to 6 terms, and its far terms are the slow ones (w(z) by the
    // continued fraction): fewer lanes.
    constexpr int W = (KIND == 0) ? 6 : 15;
    {
      const int l = lane <= 2 * W ? lane : 0;  // the rest repeat the centre
      eval(l <= W ? l : W - l, ce0, l <= W ? l : l - W);
    }
    int got = take(0, W, 0);
    if (got < 0) return got;
    int next = 1;  // the second side's next offset
    cplx last = ce0;
    if (got) {
      got = take(W + 1, 2 * W, 1);
      if (got < 0) return got;
      next = W + 1;
      last = mk(__shfl_sync(0xffffffffu, ce.re, 2 * W), __shfl_sync(0xffffffffu, ce.im, 2 * W));
    } else {
      cplx l0 = mk(__shfl_sync(0xffffffffu, ce.re, W), __shfl_sync(0xffffffffu, ce.im, W));
      for (int o = W + 1; !got; o += 32) {
        eval(o + lane, l0, lane + 1);
        got = take(0, 31, o);
        if (got < 0) return got;
        l0 = mk(__shfl_sync(0xffffffffu, ce.re, 31), __shfl_sync(0xffffffffu, ce.im, 31));
      }
      got = 0;
    }
    for (; !got; next += 32) {
      eval(-(next + lane), last, lane + 1);
      got = take(0, 31, next);
      if (got < 0) return got;
      last = mk(__shfl_sync(0xffffffffu, ce.re, 31), __shfl_sync(0xffffffffu, ce.im, 31));
    }
#pragma unroll
    for (int i = 0; i < 8; i++) S.v[i] = __shfl_sync(0xffffffffu, mine, i);
    bool rstop = true;
    if (dir != 0) {
      if (KIND == 0) {
        rstop = qp_comp(S.S(), old.S(), eps);
        if (MODE == QP_BOTH) rstop = rstop && qp_comp(S.d(0), old.d(0), eps) && qp_comp(S.d(1), old.d(1), eps);
      } else {
        rstop = false;
        if (KIND == 2 || flg == 0) {
          rstop = qp_comp(S.d(2), old.d(2), eps);
          if (MODE == QP_BOTH) rstop = rstop && qp_comp(S.S(), old.S(), eps);
        }
      }
    }
    if (rstop) {
      if (dir == 2) break;
      dir++;
      n = (dir == 1) ? nc + 1 : nc - 1;
    } else {
      n += (dir == 1) ? 1 : -1;
      if (n - nc >= LIMIT || n - nc <= -LIMIT) return ELIM;
    }
  }
  out = S;
  return cc;
}

template <int MODE>
__device__ __noinline__ int qw_serial(const QPLattice& L, const double* r, QPVal& out)
{
  return qpgf_eval<MODE>(L, r, out);
}

// a * s rounded by itself (the serial sums' results are stored before they are added up)
__device__ __forceinline__ cplx qw_scale(cplx a, double s) { return mk(__dmul_rn(a.re, s), __dmul_rn(a.im, s)); }

// The whole evaluation (qpgf_eval<MODE>), every lane with the result.
template <int MODE>
__device__ __forceinline__ int qpgf_eval_warp(const QPLattice& L, const double* r_in, int lane, QwBatch& B, QPVal& out)
{
  const double eps = QP_MEPS;
  if (r_in[2] * r_in[2] < SMT_ZPLANE * SMT_ZPLANE * fabs(L.detd)) return qw_serial<MODE>(L, r_in, out);
  const int l1 = (int)floor((r_in[0] * L.d2y - r_in[1] * L.d2x) * L.idd + 0.5);
  const int l2 = (int)floor(-(r_in[0] * L.d1y - r_in[1] * L.d1x) * L.idd + 0.5);
  const double r[3] = {r_in[0] - (double)l1 * L.d1x - (double)l2 * L.d2x, r_in[1] - (double)l1 * L.d1y - (double)l2 * L.d2y,
                       r_in[2]};
  bool use_fd = false;
  if (!L.ew_only)
    use_fd = (L.bN / L.bNp * exp(-L.bNp * fabs(r[2])) < eps) && (L.bN / L.bNm * exp(-L.bNm * fabs(r[2])) < eps);
  const double aidd = fabs(L.idd);
  int err;
  QwSum s;
  if (use_fd) {
    err = qw_sum<MODE, 2>(L, r, 0.0, eps, lane, B, s);
    if (err < 0) return err - 10;
    const double c = 0.5 * aidd;
    out.G = mul_i(qw_scale(s.S(), c));
    out.dG[0] = qw_scale(s.d(0), -c);
    out.dG[1] = qw_scale(s.d(1), -c);
    out.dG[2] = qw_scale(s.d(2), -c * r[2] / fabs(r[2]));
  } else {
    double veps = L.veps0;
    const double r2 = r[0] * r[0] + r[1] * r[1] + r[2] * r[2];
    if (L.k * L.k * veps * veps - r2 / (4.0 * veps * veps) > QP_EW_EXPM)
      veps = sqrt(QP_EW_EXPM + sqrt(L.k * L.k * r2 + QP_EW_EXPM * QP_EW_EXPM)) / (sqrt(2.0) * L.k);
    const int c1 = qw_sum<MODE, 0>(L, r, veps, eps, lane, B, s);
    if (c1 < 0) return c1 - 20;
    const double f4p = 4.0 * QP_PI;
    out.G = mk(s.v[0] / f4p, s.v[1] / f4p);
    out.dG[0] = mk(s.v[2] / -f4p, s.v[3] / -f4p);
    out.dG[1] = mk(s.v[4] / -f4p, s.v[5] / -f4p);
    out.dG[2] = qw_scale(s.d(2), -r[2] / f4p);
    const int c2 = qw_sum<MODE, 1>(L, r, veps, eps, lane, B, s);
    if (c2 < 0) return c2 - 20;
    const double c = 0.25 * aidd;
    out.G += mul_i(qw_scale(s.S(), c));
    out.dG[0] += qw_scale(s.d(0), -c);
    out.dG[1] += qw_scale(s.d(1), -c);
    out.dG[2] += qw_scale(s.d(2), c);
    err = c1 + c2;
  }
  if (l1 != 0 || l2 != 0) {
    const cplx cf = expi(-(L.vkx * ((double)l1 * L.d1x + (double)l2 * L.d2x) + L.vky * ((double)l1 * L.d1y + (double)l2 * L.d2y)));
    out.G = out.G * cf;
    for (int i = 0; i < 3; i++) out.dG[i] = out.dG[i] * cf;
  }
  return err;
}
