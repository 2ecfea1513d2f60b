// Host build of the tabulated smooth remainder of the quasi-periodic Green's function (csrc/smooth.cuh):
// a domain's plan and table on the CPU, and one pair by it and by the plain lattice sums.
#include <math.h>
#include <string.h>

#include <complex>
#include <vector>

#include "ewald_warp.cuh"
#include "self.cuh"
#include "smooth.cuh"

namespace {
struct Domain {
  QPLattice L;
  std::vector<QPProp> prop;
  SmoothPlan P;
  std::vector<cplx> tab;
  std::vector<char> have;
  SmoothLat S;
};
Domain D;

void centre_coefs(int slot)
{
  SmoothPlan& P = D.P;
  if (D.have[slot]) return;
  D.have[slot] = 1;
  SmoothCell c;
  smooth_centre(D.L, P, slot % P.N1 - P.I, slot / P.N1 % P.N2 - P.J, slot / P.N1 / P.N2, c);
  std::vector<cplx> smp(P.nth * P.nph), a(P.nth), b(P.nth);
  std::vector<double> pts(3 * P.nth * P.nph);
  for (int p = 0; p < P.nth * P.nph; p++) {
    smooth_sample_point(P, c, p, &pts[3 * p]);
    smp[p] = smooth_real(D.L, D.S, c, &pts[3 * p]);
  }
  for (int t = 0; t < P.nth; t++)  // a theta's samples share their height
    for (int a = 0; a < D.S.no1; a++)
      for (int b = 0; b < D.S.no2; b++) {
        double ax, ay;
        const cplx f = smooth_order(D.L, D.S, D.S.o1 + a, D.S.o2 + b, fabs(pts[3 * t * P.nph + 2]), &ax, &ay);
        if (f.re == 0.0 && f.im == 0.0) continue;
        for (int q = t * P.nph; q < (t + 1) * P.nph; q++) smp[q] += f * expi(ax * pts[3 * q] + ay * pts[3 * q + 1]);
      }
  cplx* al = D.tab.data() + (size_t)slot * smt_ncoef(P.L);
  for (int m = 0; m <= P.L; m++) {
    for (int t = 0; t < P.nth; t++) smooth_azimuth(P, smp.data(), t, m, a[t], b[t]);
    for (int l = m; l <= P.L; l++) {
      cplx A = mk(0, 0), B = mk(0, 0);
      for (int t = 0; t < P.nth; t++) {
        A += a[t] * P.proj[(size_t)smt_lm(P.L, m, l) * P.nth + t];
        B += b[t] * P.proj[(size_t)smt_lm(P.L, m, l) * P.nth + t];
      }
      *al++ = A;
      if (m) *al++ = B;
    }
  }
}
typedef long double X;
void gauss(int n, X* x, X* w)
{
  for (int i = 0; i < n; i++) {
    X z = cosl(3.14159265358979323846L * (i + 0.75L) / (n + 0.5L)), d = 1;
    for (int it = 0; it < 12; it++) {
      X p = 1, q = 0;
      for (int j = 1; j <= n; j++) { const X o = q; q = p; p = ((2 * j - 1) * z * q - (j - 1) * o) / j; }
      d = n * (z * p - q) / (z * z - 1);
      z -= p / d;
    }
    x[i] = z;
    w[i] = 2 / ((1 - z * z) * d * d);
  }
}
}  // namespace

extern "C" {

// Plan of the elements 1..ne of geo; lat = k, vkx, vky, d1, d2; degree 0: the cheapest.  info: on, L,
// centres, points of the quad and triangle rules.  Returns 1 when a plan exists.
int sh_plan(const double* lat, const double* geo, int ne, double npairs, int degree, int* info)
{
  memset((void*)&D.L, 0, sizeof D.L);
  if (qp_lattice_init(D.L, lat[0], lat[1], lat[2], lat[3], lat[4], lat[5], lat[6]) != 0) return 0;
  D.prop.resize(QP_PROP_CAP);
  D.L.nprop = qp_prop_list(D.L, D.prop.data(), QP_PROP_CAP);
  D.L.prop = D.prop.data();
  SmoothLat& S = D.S;
  smooth_lattice(D.L, S);
  double he = 0, ra = 0, be = 0, lo[3] = {1e300, 1e300, 1e300}, hi[3] = {-1e300, -1e300, -1e300};
  int tri = 0;
  for (int i = 1; i <= ne; i++) {
    Elem e;
    load_elem(geo, i, e);
    smooth_extent(D.L, e, &he, &ra, &be, lo, hi);
    tri |= (e.nn == 3);
  }
  const SmoothExt X = {he, hi[2] - lo[2], hi[0] - lo[0], hi[1] - lo[1], ra, be};
  double best = 1e300;
  SmoothGrid g;
  for (int d = SMT_LMIN; d <= SMT_LMAX; d++) {
    double c;
    if (degree && d != degree) continue;
    smooth_choose(D.L, S, X, npairs, 144.0, tri, 1LL << 40, d, g, c);
    if (c < best) { best = c; *static_cast<SmoothGrid*>(&D.P) = g; }
  }
  info[0] = best < 1e300 ? D.P.on : 0;
  if (best >= 1e300) return 0;
  info[1] = D.P.L; info[2] = D.P.ncent; info[3] = D.P.nq4; info[4] = D.P.nq3;
  smooth_tables_a(D.P, 0, 1);
  smooth_tables_b(D.P, 0, 1);
  smooth_tables_c(D.P, D.L.k, 0, 1);
  D.tab.assign((size_t)D.P.ncent * smt_ncoef(D.P.L) + SMT_PAD, mk(0, 0));
  D.have.assign(D.P.ncent, 0);
  return 1;
}

// Sums G[4], H[4], F, dF0, dF1 (19 doubles, scaled as the matrices hold them) of the pair (node tn of
// element t, element s) by the n x n rule: by the plan (plain 0) or the lattice sums (plain 1).
// Returns the lowest status; in_plane: whether the plan leaves the pair to the lattice sums.
int sh_pair(const double* geo, int t, int tn, int s, int plain, int n, const double* x, const double* w, double* out,
            int* in_plane)
{
  Elem es, et;
  load_elem(geo, s, es);
  load_elem(geo, t, et);
  double v0[3], v1[3];
  node_tangents(et, tn, v0, v1);
  const double* rt = geo + (size_t)t * GEO_STRIDE + GEO_REN + 3 * tn;
  *in_plane = smooth_in_plane(D.L, es, rt[2]);
  const int npts = (es.nn == 4) ? n * n : 3 * n * n;
  AccP a;
  accp_zero(a);
  int err = 0;
  cplx ph = mk(1.0, 0.0);
  if (plain) {
    for (int q = 0; q < npts; q++) {
      double z, e, wt;
      rule_point(es.nn, n, x, w, q, z, e, wt);
      const int st = accp_point(es, D.L, rt, v0, v1, z, e, wt, a);
      if (st < 0) err = st;
    }
  } else {
    const double v[3] = {es.cr[0][0] - rt[0], es.cr[1][0] - rt[1], es.cr[2][0] - rt[2]};
    double sx, sy;
    const int sh = smooth_shift(D.L, v, &sx, &sy);
    for (int q = 0; q < npts; q++) {
      double z, e, wt;
      rule_point(es.nn, n, x, w, q, z, e, wt);
      smooth_near(es, D.L.k, rt, v0, v1, sx, sy, sh, z, e, wt, a);
    }
    for (int i = 0; i < 4; i++) { a.G[i] = a.G[i] * EL_I_FP; a.H[i] = a.H[i] * EL_I_FP; }
    const int nq = es.nn == 4 ? D.P.nq4 : D.P.nq3;
    const double* tq = es.nn == 4 ? D.P.q4 : D.P.q3;
    for (int q = 0; q < nq; q++) {
      double r[3], W[3], rad[SMT_LMAX + 2], N[4], z, e;
      point_geom(es, tq[3 * q], tq[3 * q + 1], rt, r, W);
      SmoothCell c;
      smooth_cell(D.L, D.P, r[0] + sx, r[1] + sy, fabs(r[2]), c);
      centre_coefs(c.slot);
      cplx gw, hw;
      smooth_point(es, D.L, D.P, D.tab.data(), rt, sx, sy, q, rad, 1, gw, hw, z, e);
      if (es.nn == 4) bil_N4(z, e, N);
      else { lit_N3(z, e, N); N[3] = 0.0; }
      for (int i = 0; i < 4; i++) { a.G[i] += gw * N[i]; a.H[i] += hw * N[i]; }
    }
    if (sh) ph = expi(D.L.vkx * sx + D.L.vky * sy);
  }
  cplx CC[9], dCz[9], dCe[9];
  accp_finish(es, a, CC, dCz, dCe);
  for (int i = 0; i < 8; i++) { CC[i] = CC[i] * ph; out[2 * i] = CC[i].re; out[2 * i + 1] = CC[i].im; }
  out[16] = CC[8].re; out[17] = dCz[8].re; out[18] = dCe[8].re;
  return err;
}

// G, grad G, second derivatives (20 doubles a point) by the warps' sums (lanes lanes, added up) and by the
// plain sums; returns 0 when the lattice has no such sums.
int sh_ewald(const double* lat, const double* r, int n, int lanes, double* out, double* plain)
{
  QPLattice L;
  memset((void*)&L, 0, sizeof L);
  if (qp_lattice_init(L, lat[0], lat[1], lat[2], lat[3], lat[4], lat[5], lat[6]) != 0) return 0;
  std::vector<QPProp> prop(QP_PROP_CAP);
  L.nprop = qp_prop_list(L, prop.data(), QP_PROP_CAP);
  L.prop = prop.data();
  SmoothLat S;
  smooth_lattice(L, S, EWW_EXPM);
  if (!S.ok) return 0;
  for (int i = 0; i < n; i++) {
    double sum[20] = {0.0}, px = 0.0, py = 0.0;
    EwaldVal o;
    for (int l = 0; l < lanes; l++) {
      ewald_terms<true>(L, S, r + 3 * i, l, lanes, o, &px, &py);
      const double* t = reinterpret_cast<const double*>(&o);
      for (int c = 0; c < 20; c++) sum[c] += t[c];
    }
    memcpy((void*)&o, sum, sizeof o);
    ewald_phase<true>(L, px, py, o);
    memcpy(out + 20 * i, (const void*)&o, sizeof o);
    QPVal2 v;
    if (qpgf_eval2(L, r + 3 * i, v) < 0) return 0;
    memcpy(plain + 20 * i, (const void*)&v, sizeof v);
  }
  return 1;
}

// rule_order of element s of geo for the node rt, and the 51 sums (AccI's layout: G, H, dG0, dH0, dG1, dH1
// per shape function, F, dF0, dF1) of the pair by a rule of n points per direction, in extended
// precision; size: the sums of the integrands' sizes, G, H and dG, dH.
int sh_rule(const double* geo, int s, const double* rt, const double* v0, const double* v1, double kre, double kim, int n,
            double* out, double* size)
{
  typedef std::complex<X> Z;
  std::vector<X> x(n), w(n);
  gauss(n, x.data(), w.data());
  const X s3 = sqrtl(3.0L);
  Elem e;
  load_elem(geo, s, e);
  const bool quad = e.nn == 4;
  const Z k(kre, kim), I(0, 1);
  Z sum[24] = {};
  X F[3] = {}, sz[3] = {};
  for (int q = 0; q < (quad ? n * n : 3 * n * n); q++) {
    const int part = q / (n * n), i = q / n % n, j = q % n;
    X z = x[i], t = x[j], wd = w[i] * w[j], N[4] = {};
    if (quad) {
      const X a = s3 * z, b = s3 * t;
      N[0] = (1 - a) * (1 - b) / 4; N[1] = (1 + a) * (1 - b) / 4; N[2] = (1 + a) * (1 + b) / 4; N[3] = (1 - a) * (1 + b) / 4;
    } else {
      const X a = z, b = t;
      wd *= 1 + a / 4 + b / 4;
      if (part == 0) { z = (3 + 2 * a + 2 * b + a * b) / 8; t = s3 * (b - a) / 8; }
      else if (part == 1) { z = (-3 + a - 5 * b - a * b) / 16; t = s3 * (3 + 3 * a + b + a * b) / 16; }
      else { z = (-3 - 5 * a + b - a * b) / 16; t = s3 * (-3 - a - 3 * b - a * b) / 16; }
      N[0] = (1 - 2.5L * (z + s3 * t)) / 3; N[1] = (1 + 5 * z) / 3; N[2] = (1 - 2.5L * (z - s3 * t)) / 3;
    }
    X W2 = 0, R2 = 0, RW = 0, Rv[2] = {}, Wv[2] = {};
    for (int i = 0; i < 3; i++) {
      const X W = quad ? e.cw[i][0] + z * e.cw[i][1] + t * e.cw[i][2] : (X)e.cw[i][0];
      const X r = e.cr[i][0] + z * e.cr[i][1] + t * e.cr[i][2] + (quad ? z * t * e.cr[i][3] : 0) - rt[i];
      W2 += W * W; R2 += r * r; RW += r * W;
      Rv[0] += r * v0[i]; Rv[1] += r * v1[i]; Wv[0] += W * v0[i]; Wv[1] += W * v1[i];
    }
    const X R = sqrtl(R2), a = quad ? sqrtl(W2) : 1;
    const Z u = std::exp(I * k * R) * wd, b = I * k * R - (X)1, c = k * k * R2 + (X)3 * b;
    Z f[6] = {u * a / R, b * u * RW / (R2 * R)};
    for (int j = 0; j < 2; j++) {
      f[2 + 2 * j] = b * u * Rv[j] * a / (R2 * R);
      f[3 + 2 * j] = u * (c * Rv[j] * RW / R2 - b * Wv[j]) / (R2 * R);
      F[1 + j] += wd * (3 * Rv[j] * RW / R2 - Wv[j]) / (R2 * R);
    }
    F[0] += wd * RW / (R2 * R);
    for (int j = 0; j < 6; j++)
      for (int i = 0; i < 4; i++) sum[4 * j + i] += f[j] * N[i];
    const X g = wd * a * expl(-kim * R) / R, d = std::abs(k) + 1 / R, m = quad ? 1 : fmaxl(1, sqrtl(W2));
    sz[0] += g;
    sz[1] += g * d * m;
    sz[2] += 3 * g * d * d * m;
  }
  for (int i = 0; i < 24; i++) { out[2 * i] = (double)sum[i].real(); out[2 * i + 1] = (double)sum[i].imag(); }
  for (int i = 0; i < 3; i++) { out[48 + i] = (double)F[i]; size[i] = (double)sz[i]; }
  double d2 = 0.0;
  for (int i = 0; i < 3; i++) d2 += (e.cr[i][0] - rt[i]) * (e.cr[i][0] - rt[i]);
  return rule_order(e, d2, fabs(kre) + 2.5 * fabs(kim));
}

// Piece 2 of the interior self pair of element s, node tn, by the 24-point (out) and the 64-point rule
// (ref); returns whether the 24-point rule may stand for it.
int sh_self2(const double* geo, int s, int tn, double kre, double kim, const double* xs, const double* ws, const double* xh,
             const double* wh, double* out, double* ref)
{
  SelfInfo S;
  self_setup(geo, s, tn, mk(kre, kim), S);
  for (int i = 0; i < SELF_NV; i++) out[i] = ref[i] = 0.0;
  self_int_piece2(S, xh, wh, 0, 1, out, xs, ws);
  self_int_piece2(S, xh, wh, 0, 1, ref);
  return self_log_rule(S);
}

}
