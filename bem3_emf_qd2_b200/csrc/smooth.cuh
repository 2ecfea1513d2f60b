// smooth.cuh -- the quasi-periodic Green's function of the assembly as its nearest image plus a
// smooth remainder, host+device.
//
// For the points of one (collocation node, source element) pair the lattice sum splits as
//
//   G(r) = g0(r) + sum over 3 more images g0(r + R) + S(r),     g0(r) = e^{ik|r|} / (4 pi |r|),
//
// r reduced to the cell around the origin by the element's centre.  Only g0(r) varies quickly over
// the element: it keeps the rule of the pair (12 x 12, 64 x 64 or polar points) and costs one
// complex exponential a point.  The other three images of the point's 2 x 2 block and S are smooth
// there (their nearest singularity is about a lattice period away), so they are integrated with the
// few Gauss points that a smooth integrand of that size needs (smooth_nq), and S is not summed at
// all: it solves Helmholtz's equation, so on a ball around a centre c of a grid over the cell it is
//
//   S(c + d) = sum_{l <= L} f_l(|d|) sum_m [A_lm Re + B_lm Im] R_lm(d)
//
// with (L + 1)^2 complex coefficients per centre (f_l(r) = j_l(k r) / r^l, R_lm the solid harmonics), where polynomials of the same degree would need (L+1)(L+2)(L+3)/6.  The coefficients
// come from 2 (L + 1)^2 values of S on a sphere around c (Gauss-Legendre in cos(theta), equal steps
// in phi).  Those values are Ewald sums with ONE split parameter and fixed sets of terms for the whole
// table: the spheres of a layer of centres share their heights, so an order's height function is
// evaluated once per height, and over the centres of the layer the sum over the orders is a Fourier
// transform in two steps.  The parameter is small (k veps <= 1, where the per-point sums allow
// sqrt(3)), so that no term is larger than e times the sum: the table's values are more accurate than
// the per-point sums.  A point costs ~14 (L + 1)^2 multiply-adds instead of the ~200
// lattice terms of ~130 operations each; L and the grid are chosen per domain by the smaller sum of
// table and evaluation costs (smooth_plan).
//
// Two cases stay with the full lattice sums point by point: domains where the table would cost more
// than it saves, and pairs whose element lies in the plane of the node (|z| < SMT_ZPLANE periods):
// there the reference's stop rule compares z derivatives that are rounding noise, its sums stop at
// 60 to 126 terms depending on the last bits, and only the same sums give the same values.
#pragma once

#include "elem.cuh"

#define SMT_LMIN 8
#define SMT_LMAX 18
#define SMT_NQMAX 16
#define SMT_ZPLANE 1e-11
#define SMT_PMAX (SMT_NQMAX * (SMT_NQMAX + 1))
#define SMT_TOL 1e-16   // truncation of the expansions
#define SMT_QTOL 5e-16  // worst-direction error of the smooth rules
#define SMT_EXPM 1.0     // bound of (k veps)^2 of the table's Ewald sums
#define SMT_CUT 38.5     // their terms below e^-38.5 = 2e-17 are left out
#define SMT_NNEAR 21
#define SMT_TNEAR 0.5    // R / (2 ve) up to which `near` is used (its next term is below 1e-17 of the first)
#define SMT_ORDERS 5000  // most spectral orders (of the rectangle that holds them) of a table: shared memory

// c_lm = ((l - 1)^2 - m^2) / ((2l - 1)(2l - 3)) of the monic recurrence
// R_l^m = z R_{l-1}^m - c_lm r^2 R_{l-2}^m, R_m^m = (x + iy)^m, R_{m-1}^m = 0.
struct SmtRec {
  double c[SMT_LMAX + 2][SMT_LMAX + 2];  // [m][l]
  double inv[2 * SMT_LMAX + 32];         // 1 / i
  constexpr SmtRec() : c{}, inv{}
  {
    for (int m = 0; m < SMT_LMAX + 2; m++)
      for (int l = 0; l < SMT_LMAX + 2; l++)
        c[m][l] = (l >= m + 2) ? ((l - 1.0) * (l - 1.0) - 1.0 * m * m) / ((2.0 * l - 1.0) * (2.0 * l - 3.0)) : 0.0;
    for (int i = 1; i < 2 * SMT_LMAX + 32; i++) inv[i] = 1.0 / i;
  }
};
#if defined(__CUDACC__)
__device__ __constant__ SmtRec smt_rec = SmtRec();
#else
static const SmtRec smt_rec = SmtRec();
#endif

// What the plan needs from the lattice alone (host): distances, and the table's Ewald split.
struct SmoothLat {
  int ok;
  cplx e1, e2;   // Bloch phases e^{i k||.d1}, e^{i k||.d2}
  double dimg;   // distance from the cell to the nearest image other than the origin
  double dblk;   // ... to the nearest image outside a point's 2 x 2 block
  double terms;  // lattice terms of one full evaluation (estimate)
  double ve, rmax;     // split parameter; reach of the real-space terms
  int m1, m2;          // images |p| <= m1, |q| <= m2 hold that reach around every table point
  int o1, o2, no1, no2;  // spectral orders o1 .. o1 + no1 - 1, o2 .. o2 + no2 - 1
  double near[SMT_NNEAR];  // an image's real-space term without the image itself, by powers of R / (2 ve)
};

// A domain's grid of expansion centres and sampling sphere, and their tables (device memory, written
// by the plan kernel before every assembly).
struct SmoothGrid {
  int on;                 // 0: this domain is summed point by point
  int L, nth, nph;        // degree; the sphere's points nth x nph
  int n1, n2;             // grid cells per lattice vector
  int I, J, N1, N2, N3;   // centres (i / n1) d1 + (j / n2) d2 + m hz z, |i| <= I, |j| <= J, 0 <= m < N3
  int ncent;
  int nq4, nq3;           // points of the smooth rules (quads, triangles)
  double hz, rs;          // vertical spacing; sphere radius
  double rn1, rn2, rhz;   // 1 / n1, 1 / n2, 1 / hz
  double top;             // k^{L+1} / (2L+3)!!
  cplx e1, e2;            // the lattice's Bloch phases
};
struct SmoothPlan : SmoothGrid {
  double cth[SMT_LMAX + 1], sth[SMT_LMAX + 1], wth[SMT_LMAX + 1];
  double cph[2 * SMT_LMAX + 2], sph[2 * SMT_LMAX + 2];  // cos, sin of 2 pi i / nph
  double c00;                            // coefficient (0, 0) of a sample value constant over the sphere, 1 / f_0(rs)
  double q4[3 * SMT_NQMAX * SMT_NQMAX];  // zeta, eta, weight
  double q3[3 * SMT_PMAX];
  double proj[(SMT_LMAX + 1) * (SMT_LMAX + 2) / 2 * (SMT_LMAX + 1)];  // [(m, l)][theta node]
};

// Geometry that sizes the plan: the largest half edge, the extent of the elements in z and in the
// lattice's fractional coordinates, the elements' radius and how much their normals turn.
struct SmoothExt {
  double half_edge, zlen, ulen, vlen, radius;
  double bend;  // largest variation of the normal over an element, |W(+-1)  - W(0)| / |W(0)| (quads)
};

// Coefficients of a centre, (L + 1)^2, and one more for even L: with the device table's first at an odd
// place then (smt_at), every pair A, B of m >= 1 is one aligned 32-byte load.
BEM_HD int smt_ncoef(int L) { return (L + 1) * (L + 1) + !(L & 1); }
template <class T>
BEM_HD T* smt_at(T* tab, int L, int slot)
{
#if defined(__CUDA_ARCH__)
  tab += !(L & 1);
#endif
  return tab + (size_t)slot * smt_ncoef(L);
}
// position of (m, l) in the coefficient order: m = 0: l = 0..L; then m = 1: l = 1..L; ...
BEM_HD int smt_lm(int L, int m, int l) { return m * (L + 1) - m * (m - 1) / 2 + (l - m); }

// expm: bound of (k veps)^2 of the sums.
inline void smooth_lattice(const QPLattice& L, SmoothLat& S, double expm = SMT_EXPM)
{
  S.ok = 0;
  S.dimg = S.dblk = S.terms = S.ve = S.rmax = 0.0;
  S.m1 = S.m2 = S.o1 = S.o2 = S.no1 = S.no2 = 0;
  if (!(L.k > 0.0)) return;
  // squared distances at a 9 x 9 grid of the cell's points (corners and edges among them)
  double d0 = 1e300, db = 1e300;
  for (int a = -4; a <= 4; a++)
    for (int b = -4; b <= 4; b++) {
      const double u = 0.125 * a, v = 0.125 * b;
      const double x = u * L.d1x + v * L.d2x, y = u * L.d1y + v * L.d2y;
      for (int p = -3; p <= 3; p++)
        for (int q = -3; q <= 3; q++) {
          if (p == 0 && q == 0) continue;
          const double X = x + p * L.d1x + q * L.d2x, Y = y + p * L.d1y + q * L.d2y;
          const double d = X * X + Y * Y;
          d0 = fmin(d0, d);
          // the block of a point: images 0 and -sign(u), 0 and -sign(v); u or v = 0 may have either
          const int inu = p == 0 || (p == -1 && a > 0) || (p == 1 && a < 0);
          const int inv = q == 0 || (q == -1 && b > 0) || (q == 1 && b < 0);
          if (!(inu && inv)) db = fmin(db, d);
        }
    }
  S.e1 = expi(L.vkx * L.d1x + L.vky * L.d1y);
  S.e2 = expi(L.vkx * L.d2x + L.vky * L.d2y);
  S.dimg = sqrt(d0);
  S.dblk = sqrt(db);
  // Ewald terms of a per-point sum, at the split parameter the clamp gives near the origin
  double ve = sqrt(QP_EW_EXPM) / L.k;
  if (ve > L.veps0) ve = L.veps0;
  const double am2 = 37.0 / (ve * ve) + L.k * L.k, R = 2.0 * ve * 6.1, det = fabs(L.detd);
  S.terms = det / (4.0 * QP_PI) * am2 + QP_PI * R * R / det + 30.0;
  // the table's sums
  S.ve = sqrt(expm) / L.k;
  if (S.ve > L.veps0) S.ve = L.veps0;
  S.rmax = 2.0 * S.ve * sqrt(SMT_CUT + L.k * L.k * S.ve * S.ve);
  // v(R) - cos kR of smooth_real, over R / (2 ve) = t: with v = Re e^{-ikR} erfc(t - i k ve) it is F(t) =
  // -Re e^{-ikR} erf(t - i k ve), which solves F' = 2 k ve D - (2 / sqrt(pi)) e^{(k ve)^2 - t^2},
  // D' = -2 k ve F, F(0) = 0, D(0) = erfi(k ve).
  {
    const double ke = L.k * S.ve, g0 = 2.0 * QP_INV_SQRTPI * exp(ke * ke);
    double D = 0.0, term = ke, F = 0.0, E[2] = {1.0, 0.0};
    for (int m = 0; m < 60; m++) {
      D += term / (2 * m + 1);
      term *= ke * ke / (m + 1);
    }
    D *= 2.0 * QP_INV_SQRTPI;
    for (int n = 0; n < SMT_NNEAR; n++) {
      const double f = (2.0 * ke * D - g0 * E[n & 1]) / (n + 1);
      D = -2.0 * ke * F / (n + 1);
      E[n & 1] *= -2.0 / (n + 2);
      S.near[n] = F = f;
    }
  }
  const double l1 = sqrt(L.d1x * L.d1x + L.d1y * L.d1y), l2 = sqrt(L.ad22);
  // table points: within half a cell, an element's radius (0.46 dimg at most with a smooth rule), half a
  // grid cell's diagonal and the sampling sphere's radius (smooth_choose) of the origin
  const double ext = 0.46 * S.dimg + (0.145 + 0.29) * S.dblk;
  const double b1 = S.rmax * l2 / det + fmax(1.5, 0.5 + ext * l2 / det), b2 = S.rmax * l1 / det + fmax(1.5, 0.5 + ext * l1 / det);
  const double amax = sqrt(SMT_CUT / (S.ve * S.ve) + L.k * L.k);
  const double c1 = (L.vkx * L.d1x + L.vky * L.d1y) / (2.0 * QP_PI), c2 = (L.vkx * L.d2x + L.vky * L.d2y) / (2.0 * QP_PI);
  const double w1 = amax * l1 / (2.0 * QP_PI), w2 = amax * l2 / (2.0 * QP_PI);
  if (!(b1 < 40.0 && b2 < 40.0 && w1 < 1000.0 && w2 < 1000.0)) return;
  S.m1 = (int)b1; S.m2 = (int)b2;
  S.o1 = (int)ceil(c1 - w1); S.o2 = (int)ceil(c2 - w2);
  S.no1 = (int)floor(c1 + w1) - S.o1 + 1; S.no2 = (int)floor(c2 + w2) - S.o2 + 1;
  if (S.no1 < 1 || S.no2 < 1 || S.no1 > 128 || S.no2 > 128 || S.no1 * S.no2 > SMT_ORDERS) return;
  // a grazing order (beta_n = 0): the lattice sums report it
  for (int a = 0; a < S.no1; a++)
    for (int b = 0; b < S.no2; b++) {
      const double ax = -L.vkx + (S.o1 + a) * L.g1x + (S.o2 + b) * L.g2x;
      const double ay = -L.vky + (S.o1 + a) * L.g1y + (S.o2 + b) * L.g2y;
      if (fabs(L.k * L.k - ax * ax - ay * ay) < 1e-13 * L.k * L.k) return;
    }
  S.ok = 1;
}

// Gauss points per direction for the images on an element whose half edges are at most 1, the nearest q away
// from its middle: the rule's error is below SMT_QTOL of the integrand's size, for 1 / R and r / R^3 times the shape
// functions, rows up to 1 nearer than the middle, in the worst direction (extended precision; squares and rhombi
// down to 45 degrees; triangles, whose rule has n + 1 by n points: equilateral to 150 degrees, and slivers).
BEM_HD int smooth_nq_image(double q, int tri)
{
  if (q >= (tri ? 83.0 : 91.0)) return 4;
  if (q >= (tri ? 27.0 : 30.1)) return 5;
  if (q >= (tri ? 13.3 : 14.6)) return 6;
  if (q >= (tri ? 8.25 : 9.05)) return 7;
  if (q >= (tri ? 5.85 : 6.45)) return 8;
  if (q >= (tri ? 4.55 : 5.05)) return 9;
  if (q >= (tri ? 3.75 : 4.28)) return 10;
  if (q >= (tri ? 3.22 : 3.75)) return 11;
  if (q >= (tri ? 2.85 : 3.38)) return 12;
  if (q >= (tri ? 2.58 : 3.10)) return 13;
  if (q >= (tri ? 2.38 : 2.90)) return 14;
  if (q >= (tri ? 2.22 : 2.75)) return 15;
  return q >= (tri ? 2.09 : 2.63) ? 16 : 0;
}
// Gauss points per direction for a smooth integrand on an edge of half length h: a wave of number k and
// images at distance d (smooth_nq_image), times the (linear) shape functions, and the area factor |W| of an
// element whose normal turns by `bend`.  The error of the n-point rule is K_n f^{(2n)} h^{2n} / (2n)!,
// K_n = 2^{2n} (n!)^4 / ((2n+1) ((2n)!)^2) (mean over the edge); |W| = |W0| sqrt(1 + bend^2 x^2) has the
// Taylor coefficient binom(1/2, n) bend^{2n} ~ bend^{2n} / (2 sqrt(pi) n^{3/2}).  The smallest n whose errors,
// for the worst direction, stay below SMT_QTOL; 0 when SMT_NQMAX points do not reach it.
BEM_HD int smooth_nq(double k, double h, double d, double bend, int tri = 0)
{
  const double x = k * h;
  const int ni = smooth_nq_image(d / h, tri);
  if (ni == 0) return 0;
  const double lb = log(bend > 1e-9 ? bend : 1e-9), lx = log(x);
  double lf = 0.0;   // ln n!
  double lf2 = 0.0;  // ln (2n)!
  for (int n = 1; n <= SMT_NQMAX; n++) {
    lf += log((double)n);
    lf2 += log((double)(2 * n - 1)) + log((double)(2 * n));
    if (n < ni) continue;
    const double K = (2 * n) * 0.6931471805599453 + 4.0 * lf - log(2.0 * n + 1.0) - 2.0 * lf2;
    const double e1 = exp(K - lf2 + (2 * n - 1) * lx) * (x + 2 * n);
    const double e3 = exp(K + 2 * n * lb) * 0.29 / (n * sqrt((double)n));
    if (e1 <= SMT_QTOL && e3 <= SMT_QTOL) return n;
  }
  return 0;
}

// Largest ball of an expansion of degree L: the first neglected wave (k a)^{L+1} / (2L+1)!! and the
// first neglected power of the images at distance d, (a / d)^{L+1}, both at SMT_TOL.
BEM_HD double smooth_radius(int L, double k, double d)
{
  double df = 0.0;
  for (int l = 1; l <= L; l++) df += log(2.0 * l + 1.0);
  const double lt = log(SMT_TOL);
  const double a1 = exp((df + lt) / (L + 1)) / k;
  const double a2 = d * exp(lt / (L + 1));
  double a = a1 < a2 ? a1 : a2;
  if (k * a > 2.5) a = 2.5 / k;  // below the first zero of every j_l
  return a;
}

// Grid of centres for balls of radius a: near-cubic cells whose half diagonal is at most a.
// Returns the number of centres (0: none fits); fills n1, n2, I, J, N3, hz.
BEM_HD double smooth_grid(const QPLattice& L, const SmoothExt& X, double a, SmoothGrid& P)
{
  const double l1 = sqrt(L.d1x * L.d1x + L.d1y * L.d1y), l2 = sqrt(L.ad22);
  double h = 2.0 * a / sqrt(3.0);
  for (int it = 0; it < 12; it++, h *= 0.93) {
    const double m1 = ceil(l1 / h), m2 = ceil(l2 / h);
    if (m1 > 400.0 || m2 > 400.0) return 0.0;
    const double ax = L.d1x / m1, ay = L.d1y / m1, bx = L.d2x / m2, by = L.d2y / m2;
    const double dp = (ax + bx) * (ax + bx) + (ay + by) * (ay + by), dm = (ax - bx) * (ax - bx) + (ay - by) * (ay - by);
    const double dd = dp > dm ? dp : dm;
    const double hz2 = 4.0 * a * a - dd;
    if (!(hz2 > 0.25 * h * h)) continue;
    double hz = sqrt(hz2);
    if (hz > 1.5 * h) hz = 1.5 * h;
    // fractional reach of the points: the reduced centre's, plus the element's radius
    const double det = fabs(L.detd);
    const double ru = X.radius * l2 / det, rv = X.radius * l1 / det;
    if (!(ru < 2.0 && rv < 2.0 && X.zlen < 1e4 * hz)) return 0.0;
    const double u = fmin(0.5, X.ulen) + ru, v = fmin(0.5, X.vlen) + rv;
    P.n1 = (int)m1; P.n2 = (int)m2;
    P.I = (int)ceil(u * m1 - 0.5 + 1e-9); P.J = (int)ceil(v * m2 - 0.5 + 1e-9);
    P.N1 = 2 * P.I + 1; P.N2 = 2 * P.J + 1;
    P.hz = hz;
    P.N3 = (int)ceil(X.zlen / hz - 0.5 + 1e-9) + 1;
    return (double)P.N1 * P.N2 * P.N3;
  }
  return 0.0;
}

// Time of a degree-L plan in ps of one B200, fitted to the kernels' times (CUPTI) at degrees 9 to 18 for 24 to 864
// quads, periods over wavelengths 1.2 to 3.75 (63 points, 0.2 to 52 ms): the evaluations at the pairs' smooth points
// (k_reg_smooth; within 10 % above 0.7 ms), and the table's samples: the transform's orders and its two steps
// (k_smooth_spectral, 30 %), the real-space terms within reach and the images (k_smooth_project, 20 % above
// 0.1 ms).  A plan for 384 quads at 0.63: degree 12 8.5 ms, 11 9.2, 13 8.7; a count of operations without the
// kernels' rates preferred 11 and below.
BEM_HD double smooth_cost(const SmoothLat& S, const SmoothGrid& P, double det, double pts, int L)
{
  const double ns = 2.0 * (L + 1) * (L + 1), o1 = S.no1, o2 = S.no2;
  const double real = QP_PI * S.rmax * S.rmax / det * 111.0 + 41.0;
  const double spec = 2.4 * o1 * o2 * P.N2 + 0.94 * o1 * P.N1 * P.N2 + 8.2 * o1 * o2;
  // fewer than 640 centres take no less: one centre's samples by its CTA (722 of them 162 us)
  return pts * (0.96 * smt_ncoef(L) + 104.0) + ns * (fmax((double)P.ncent, 640.0) * real + P.N3 * spec);
}
// ... of one lattice sum point by point, per term (k_reg_periodic: 10 to 18 from 1,090 to 160 terms)
#define SMT_TERM_PS 14.0

// f_l(r) = j_l(k r) / r^l for l = 0 .. L + 1 into out[l * st], r2 = r^2 (k r <= 2.5): the top two from
// the series j_l(x) = x^l / (2l+1)!! (1 - x^2 / (2 (2l+3)) + ...), the rest by f_{l-1} = ((2l+1) f_l -
// k r^2 f_{l+1}) / k.  top = k^{L+1} / (2L+3)!!.
BEM_HD void smooth_radial(double k, double r2, int L, double top, double* out, int st)
{
  const double t = -0.5 * k * k * r2, ik = 1.0 / k;
  double f[2];
  for (int q = 0; q < 2; q++) {
    const int l = L + 1 - q;
    double s = 1.0, term = 1.0;
    for (int i = 1; i <= 12; i++) {
      term *= t * smt_rec.inv[i] * smt_rec.inv[2 * l + 2 * i + 1];
      s += term;
      if (fabs(term) < 1e-18) break;
    }
    f[q] = s * top;
    top *= (2.0 * L + 3.0) * ik;
  }
  double hi = f[0], lo = f[1];
  out[(L + 1) * st] = hi;
  out[L * st] = lo;
  const double kr2 = k * r2;
  for (int l = L; l >= 1; l--) {
    const double n = ((2.0 * l + 1.0) * lo - kr2 * hi) * ik;
    hi = lo;
    lo = n;
    out[(l - 1) * st] = n;
  }
}

// Coefficient i of a centre (16-byte load; the table is 256-byte aligned).
BEM_HD cplx smt_ld(const cplx* __restrict__ al, int i)
{
#if defined(__CUDA_ARCH__)
  const double2 v = __ldg(reinterpret_cast<const double2*>(al) + i);
  return mk(v.x, v.y);
#else
  return al[i];
#endif
}

// Coefficients i, i + 1 by one 32-byte load.
BEM_HD void smt_ld2(const cplx* __restrict__ al, int i, cplx& A, cplx& B)
{
#if defined(__CUDA_ARCH__)
  asm("ld.global.nc.v4.f64 {%0, %1, %2, %3}, [%4];" : "=d"(A.re), "=d"(A.im), "=d"(B.re), "=d"(B.im) : "l"(al + i));
#else
  A = al[i]; B = al[i + 1];
#endif
}

// S and W . grad S at the offset (x, y, z) from a centre, from its coefficients al; rad as
// smooth_radial fills it.  The coefficients are one stream; the next pair of it is loaded a
// step ahead (up to 2 past the centre's: the table has SMT_PAD more).
#define SMT_PAD 4
BEM_HD void smooth_eval(const cplx* __restrict__ al, int L, double k, double x, double y, double z, double Wx, double Wy,
                        double Wz, const double* rad, int st, cplx& S, cplx& D)
{
  const double r2 = x * x + y * y + z * z;
  const double wd = Wx * x + Wy * y + Wz * z;
  const double wd2 = 2.0 * wd, kw = -k * wd;  // d f_l / dr = -k r f_{l+1}
  double Sr = 0.0, Si = 0.0, Dr = 0.0, Di = 0.0;
  cplx A = smt_ld(al, 0);
  {  // m = 0: R_l^0, its derivative along W; v, u: value and derivative times f_l
    double a = 1.0, d = 0.0, b = 0.0, e = 0.0;
    double j = rad[0];
    for (int l = 0; l <= L; l++) {
      const cplx An = smt_ld(al, l + 1);
      const double jn = rad[(l + 1) * st];
      const double v = j * a, u = j * d + (kw * jn) * a;
      Sr += A.re * v; Si += A.im * v; Dr += A.re * u; Di += A.im * u;
      const double c = smt_rec.c[0][l + 1], t1 = c * r2, t2 = c * wd2;
      const double na = fma(z, a, -(t1 * b)), nd = fma(z, d, fma(Wz, a, -fma(t2, b, t1 * e)));
      b = a; e = d; a = na; d = nd;
      j = jn;
      A = An;
    }
  }
  al += L + 1;
  cplx B;
  smt_ld2(al, 0, A, B);
  // m >= 1: R_l^m = q_l (x + i y)^m with q_l real.  Per m the sums over l of f_l q_l and of its derivative
  // along W, times A and times B; the power of x + i y and its derivative come in once per m.
  double pr = x, pi = y, qr = Wx, qi = Wy;  // (x + i y)^m and its derivative along W
  for (int m = 1; m <= L; m++) {
    double a = 1.0, d = 0.0, b = 0.0, e = 0.0;
    double VAr = 0.0, VAi = 0.0, VBr = 0.0, VBi = 0.0, UAr = 0.0, UAi = 0.0, UBr = 0.0, UBi = 0.0;
    const double* rl = rad + m * st;
    const double* rc = &smt_rec.c[m][m + 1];
    double j = rl[0];
    // one degree: adds the terms of q_l = a, then b becomes q_{l+1}
    auto step = [&](double& a, double& d, double& b, double& e) {
      al += 2;
      cplx An, Bn;
      smt_ld2(al, 0, An, Bn);
      rl += st;
      const double jn = *rl;
      const double v = j * a, u = j * d + (kw * jn) * a;
      VAr += A.re * v; VAi += A.im * v; VBr += B.re * v; VBi += B.im * v;
      UAr += A.re * u; UAi += A.im * u; UBr += B.re * u; UBi += B.im * u;
      const double c = *rc++, t1 = c * r2, t2 = c * wd2;
      // the newest values (d, a) come in last: a step's dependent chain is two operations
      e = fma(z, d, fma(Wz, a, -fma(t2, b, t1 * e)));
      b = fma(z, a, -(t1 * b));
      j = jn;
      A = An; B = Bn;
    };
    int l = m;
    for (; l < L; l += 2) {
      step(a, d, b, e);
      step(b, e, a, d);
    }
    if (l == L) step(a, d, b, e);
    Sr += VAr * pr + VBr * pi; Si += VAi * pr + VBi * pi;
    Dr += UAr * pr + UBr * pi + VAr * qr + VBr * qi;
    Di += UAi * pr + UBi * pi + VAi * qr + VBi * qi;
    const double nr = pr * x - pi * y, ni = pr * y + pi * x;
    const double mr = qr * x - qi * y + pr * Wx - pi * Wy, mi = qr * y + qi * x + pr * Wy + pi * Wx;
    pr = nr; pi = ni; qr = mr; qi = mi;
  }
  S = mk(Sr, Si);
  D = mk(Dr, Di);
}

// g0 and W . grad g0 at r.
BEM_HD void smooth_image(double k, double x, double y, double z, double Wx, double Wy, double Wz, cplx& g, cplx& h)
{
  const double r2 = x * x + y * y + z * z;
  const double i_r = rsqrt_(r2);
  const double kr = k * r2 * i_r;
  g = expi(kr) * (EL_I_FP * i_r);
  h = (g * mk(-1.0, kr)) * ((Wx * x + Wy * y + Wz * z) * i_r * i_r);
}

// Centre of the grid cell that holds r: indices, and the position.
struct SmoothCell {
  int slot;
  double cx, cy, cz;
  double su, sv;  // the other images of the block are r + su d1, r + sv d2, r + su d1 + sv d2
};
BEM_HD void smooth_centre(const QPLattice& L, const SmoothPlan& P, int i, int j, int m, SmoothCell& c)
{
  c.slot = (m * P.N2 + (j + P.J)) * P.N1 + (i + P.I);
  const double u = i * P.rn1, v = j * P.rn2;
  c.cx = u * L.d1x + v * L.d2x;
  c.cy = u * L.d1y + v * L.d2y;
  c.cz = m * P.hz;
  c.su = (i >= 0) ? -1.0 : 1.0;
  c.sv = (j >= 0) ? -1.0 : 1.0;
}
// z must be >= 0; indices are clamped to the grid (the plan's reach covers every point)
BEM_HD void smooth_cell(const QPLattice& L, const SmoothPlan& P, double x, double y, double z, SmoothCell& c)
{
  const double u = (x * L.d2y - y * L.d2x) * L.idd, v = (y * L.d1x - x * L.d1y) * L.idd;
  int i = (int)rint(u * P.n1), j = (int)rint(v * P.n2), m = (int)rint(z * P.rhz);
  i = i < -P.I ? -P.I : (i > P.I ? P.I : i);
  j = j < -P.J ? -P.J : (j > P.J ? P.J : j);
  m = m < 0 ? 0 : (m >= P.N3 ? P.N3 - 1 : m);
  smooth_centre(L, P, i, j, m, c);
}

// The smooth part of G and of W . grad G at r (every image but the nearest): the three other images
// of the block and the expansion.  tab: coefficients of every centre; rad: scratch for L + 2 values.
BEM_HD void smooth_rest(const QPLattice& L, const SmoothPlan& P, const cplx* __restrict__ tab, const double* r,
                        const double* W, double* rad, int st, cplx& g, cplx& h)
{
  // S is even in z: the table holds z >= 0
  const double sg = (r[2] < 0.0) ? -1.0 : 1.0;
  const double z = sg * r[2], Wz = sg * W[2];
  SmoothCell c;
  smooth_cell(L, P, r[0], r[1], z, c);
  const double x = r[0] - c.cx, y = r[1] - c.cy, zz = z - c.cz;
  smooth_radial(L.k, x * x + y * y + zz * zz, P.L, P.top, rad, st);
  smooth_eval(smt_at(tab, P.L, c.slot), P.L, L.k, x, y, zz, W[0], W[1], Wz, rad, st, g, h);
  const cplx p1 = c.su > 0.0 ? P.e1 : conj(P.e1), p2 = c.sv > 0.0 ? P.e2 : conj(P.e2);
#if defined(__CUDA_ARCH__)
#pragma unroll 1
#endif
  for (int q = 1; q < 4; q++) {
    const double a = (q & 1) ? c.su : 0.0, b = (q & 2) ? c.sv : 0.0;
    const double X = a * L.d1x + b * L.d2x, Y = a * L.d1y + b * L.d2y;
    cplx gi, hi;
    smooth_image(L.k, r[0] + X, r[1] + Y, z, W[0], W[1], Wz, gi, hi);
    const cplx ph = q == 1 ? p1 : q == 2 ? p2 : p1 * p2;
    g += ph * gi;
    h += ph * hi;
  }
}

// Products and sums rounded one by one (no contraction): near a grazing order k^2 - |a|^2 cancels, and
// its value must be the one that qp_prop_list computes on the host.
BEM_HD double smt_mul(double a, double b)
{
#if defined(__CUDA_ARCH__)
  return __dmul_rn(a, b);
#else
  return a * b;
#endif
}
BEM_HD double smt_add(double a, double b)
{
#if defined(__CUDA_ARCH__)
  return __dadd_rn(a, b);
#else
  return a + b;
#endif
}

// Height function of spectral order (q1, q2) of the table's sums at height z >= 0, times i / (4 |cell|):
// the order's share of G is this times e^{i a.rho}, a = (*ax, *ay).  Zero beyond the cut.  SPLIT: without
// the wave of order (0, 0) where smooth_wave_diff has it (smooth_split).
BEM_HD int smooth_split(const QPLattice& L) { return L.k * L.k * fabs(L.detd) < 1.0; }
template <bool SPLIT = false>
BEM_HD cplx smooth_order(const QPLattice& L, const SmoothLat& S, int q1, int q2, double z, double* ax, double* ay)
{
  *ax = smt_add(smt_add(-L.vkx, smt_mul(q1, L.g1x)), smt_mul(q2, L.g2x));
  *ay = smt_add(smt_add(-L.vky, smt_mul(q1, L.g1y)), smt_mul(q2, L.g2y));
  const double b2 = smt_add(smt_add(smt_mul(L.k, L.k), -smt_mul(*ax, *ax)), -smt_mul(*ay, *ay));
  const double c = 0.25 * fabs(L.idd), y = z / (2.0 * S.ve);
  if (-b2 * S.ve * S.ve > SMT_CUT || b2 == 0.0) return mk(0.0, 0.0);
  const double bn = sqrt(fabs(b2)), x = bn * S.ve;
  if (b2 > 0.0) {
    const cplx ff = expi(bn * z);
    const cplx w = faddeeva_w_upper(x, y);
    const double ef = exp(x * x - y * y), f = 2.0 * c / bn;
    if (SPLIT && q1 == 0 && q2 == 0 && smooth_split(L)) return mk(-f * ef * w.im, 0.0);
    return mk(-f * (ef * w.im + ff.im), f * ff.re);  // i c F, F = (2 / bn) (i ef Im w + ff)
  }
  const double E = exp(-(x * x + y * y));
  const double f1 = E * qp_erfcx_poly(x + y);
  const double f2 = (x >= y) ? E * qp_erfcx_poly(x - y) : 2.0 * exp(-bn * z) - E * qp_erfcx_poly(y - x);
  return mk(c * (f1 + f2) / bn, 0.0);
}

// Sample p (theta p / nph, phi p % nph) of the sphere around a centre: its point.
BEM_HD void smooth_sample_point(const SmoothPlan& P, const SmoothCell& c, int p, double* r)
{
  const int t = p / P.nph, f = p - t * P.nph;
  r[0] = c.cx + P.rs * P.sth[t] * P.cph[f];
  r[1] = c.cy + P.rs * P.sth[t] * P.sph[f];
  r[2] = c.cz + P.rs * P.cth[t];
}

// The plane wave of order (0, 0), f_0 e^{i (beta |z| + a.rho)} with f_0 = i / (2 beta |cell|): its value K at
// centre c and, for sample p, the difference from it.  Where the wavelength is far above the period this wave is
// large (1 / (2 k |cell|)) and nearly constant: its rounding in the samples, over the sphere's radius, would be
// the error of the table's gradients.  K belongs to degree 0 alone (c00), the differences are taken without
// cancellation.  Only for k^2 |cell| < 1 (smooth_split): above, the wider sphere (smooth_choose) is enough, and the
// differences would cost k_smooth_project 2 % (384 quads at 0.63: 867 -> 886 us).  H of 96 quads, period 1,
// against 64-bit sums, of a pair's largest: 4e-15 at wavelength 3 (no split), 7e-15, 6e-15 at 10, 50 (1.7e-14, 8e-14,
// 4e-13 with neither; the point-by-point sums 2e-15).
BEM_HD int smooth_wave0(const QPLattice& L, double* beta)
{
  const double b2 = smt_add(smt_add(smt_mul(L.k, L.k), -smt_mul(L.vkx, L.vkx)), -smt_mul(L.vky, L.vky));
  *beta = sqrt(fabs(b2));
  return smooth_split(L) && b2 > 0.0;
}
BEM_HD cplx smooth_wave_centre(const QPLattice& L, const SmoothCell& c)
{
  double beta;
  if (!smooth_wave0(L, &beta)) return mk(0.0, 0.0);
  return mul_i(expi(beta * c.cz - L.vkx * c.cx - L.vky * c.cy)) * (0.5 * fabs(L.idd) / beta);
}
BEM_HD cplx smooth_wave_diff(const QPLattice& L, const SmoothPlan& P, const SmoothCell& c, int p, cplx K)
{
  double beta;
  if (!smooth_wave0(L, &beta)) return mk(0.0, 0.0);
  const int t = p / P.nph, f = p - t * P.nph;
  const double dz = P.rs * P.cth[t], dx = P.rs * P.sth[t] * P.cph[f], dy = P.rs * P.sth[t] * P.sph[f];
  // |cz + dz| - cz: below the plane the wave is the mirror image
  const double d = beta * (c.cz + dz < 0.0 ? -dz - 2.0 * c.cz : dz) - L.vkx * dx - L.vky * dy;
  const cplx h = expi(0.5 * d);  // e^{id} - 1 = 2i sin(d/2) e^{id/2}
  return K * mk(-2.0 * h.im * h.im, 2.0 * h.im * h.re);
}

// Real-space part of the table's sums at r, minus the block's four images.  Within SMT_TNEAR of an image both are
// nearly 1 / R: their difference comes from its series (SmoothLat::near), without the cancellation.
BEM_HD cplx smooth_real(const QPLattice& L, const SmoothLat& S, const SmoothCell& c, const double* r)
{
  const double ke = L.k * S.ve, h = 0.5 / S.ve, c4 = EL_I_FP, z2 = r[2] * r[2], r2max = S.rmax * S.rmax;
  cplx s = mk(0.0, 0.0);
  for (int p = -S.m1; p <= S.m1; p++)
    for (int q = -S.m2; q <= S.m2; q++) {
      const double X = p * L.d1x + q * L.d2x, Y = p * L.d1y + q * L.d2y;
      const double x = r[0] + X, y = r[1] + Y, R2 = x * x + y * y + z2;
      const int img = (p == 0 || p == (int)c.su) && (q == 0 || q == (int)c.sv);
      if (!img && R2 > r2max) continue;
      const double Rc = fmax(R2, 1e-200), iR = rsqrt_(Rc), R = Rc * iR, t = R * h;
      cplx v = mk(0.0, 0.0);
      if (img && t < SMT_TNEAR) {  // close to the image: the difference of two 1 / R by its series
        double f = S.near[SMT_NNEAR - 1];
        for (int n = SMT_NNEAR - 2; n >= 0; n--) f = fma(f, t, S.near[n]);
        v = mk(f * t, -expi(L.k * R).im);
      } else {
        if (R2 <= r2max) v.re = exp(ke * ke - t * t) * faddeeva_w_upper(ke, t).re;
        if (img) v -= expi(L.k * R);
      }
      s += (expi(L.vkx * X + L.vky * Y) * v) * (c4 * iR);
    }
  return s;
}

// Azimuthal sums of one centre's samples (nth x nph, phi fastest): a, b = sum over phi of the sample
// times cos, sin of m phi at theta node t.
BEM_HD void smooth_azimuth(const SmoothPlan& P, const cplx* smp, int t, int m, cplx& a, cplx& b)
{
  cplx c = mk(0.0, 0.0), s = mk(0.0, 0.0);
  for (int f = 0, q = 0; f < P.nph; f++) {
    const cplx v = smp[t * P.nph + f];
    c += v * P.cph[q];
    s += v * P.sph[q];
    q += m;
    if (q >= P.nph) q -= P.nph;
  }
  a = c;
  b = s;
}

// Gauss-Legendre node and weight i of n on [-1, 1] (Newton on P_n).
BEM_HD void smooth_gauss(int n, int i, double& x, double& w)
{
  double z = cos(QP_PI * (i + 0.75) / (n + 0.5)), pp = 1.0;
  for (int it = 0; it < 20; it++) {
    double p1 = 1.0, p2 = 0.0;
    for (int j = 1; j <= n; j++) {
      const double p3 = p2;
      p2 = p1;
      p1 = ((2.0 * j - 1.0) * z * p2 - (j - 1.0) * p3) / j;
    }
    pp = n * (z * p1 - p2) / (z * z - 1.0);
    const double dz = p1 / pp;
    z -= dz;
    if (fabs(dz) <= 1e-16) break;
  }
  x = z;
  w = 2.0 / ((1.0 - z * z) * pp * pp);
}

// The plan's choice of degree and grid, then its tables; the tables are filled by part = 0, 1, ... of
// nparts (threads), with a barrier between the two stages (smooth_tables_a, _b).
BEM_HD void smooth_choose(const QPLattice& L, const SmoothLat& S, const SmoothExt& X, double npairs, double near, int tri,
                          long long cap, int degree, SmoothGrid& P, double& cost, double chain = 0.0)
{
  // degree L alone (the caller takes the cheapest).  tri: 1 some of the elements are triangles, 2 all.  near:
  // points of a quad's rule, three times that on a triangle; 0 where each "pair" is one point.  chain > 0: field points, a thread taking `chain` rule points in
  // turn (their latency counts: 105,000 times the rate's time for each), made without regard to the plain sums
  cost = 1e300;
  P.on = 0;
  if (!S.ok) return;
  const int n3 = tri ? smooth_nq(L.k, X.half_edge, S.dimg, X.bend, 1) : 1;
  const int n4 = tri == 2 ? n3 : smooth_nq(L.k, X.half_edge, S.dimg, X.bend);
  if (n4 == 0 || n3 == 0) return;
  const double a = smooth_radius(degree, L.k, S.dblk);
  const double nc = smooth_grid(L, X, a, P);
  if (!(nc > 0.0) || nc * smt_ncoef(degree) + SMT_PAD > (double)cap) return;
  P.L = degree;
  P.nth = degree + 1;
  P.nph = 2 * degree + 2;
  P.ncent = (int)nc;
  P.nq4 = n4 * n4;
  P.nq3 = n3 * (n3 + 1);
  const double nq = near > 0.0 ? (tri ? P.nq3 : P.nq4) : 1.0;
  const double pts = npairs * nq;
  cost = smooth_cost(S, P, fabs(L.detd), chain > 0.0 ? fmax(1.7 * pts, 1.05e5 * chain * nq) : pts, degree);
  // point by point the regular pairs' points and the self pairs' (6,144 a row, 24 in turn by a thread at 1 us a term:
  // 5.4 of the 7.6 ms of 24 quads at 0.63, where the table's way takes 0.8)
  const double points = npairs * (near > 0.0 ? (tri ? 3.0 * near : near) : 1.0) + 2.0 * sqrt(npairs) * 6144.0;
  const double plain = S.terms * fmax(SMT_TERM_PS * points, 24e6);
  if (chain > 0.0 || cost < 0.8 * plain) P.on = 1;
  P.rn1 = 1.0 / P.n1; P.rn2 = 1.0 / P.n2; P.rhz = 1.0 / P.hz;
  P.e1 = S.e1; P.e2 = S.e2;
  P.top = L.k / 3.0;
  for (int l = 1; l <= degree; l++) P.top *= L.k / (2.0 * l + 3.0);
  // The sphere: twice the grid cell's half diagonal rg, so that the samples' rounding reaches the cell damped
  // by 2^-l at degree l (over the cell's own sphere the gradients' error was L / rg times it), but well within
  // the first zero of the Bessel functions (j_0 at pi; at k rs = 3.1 the constant part's error is 15 times as large).  The neglected degrees reach the kept ones only by aliasing,
  // (rg / d)^l (rs / d)^(2 (L + 1 - l)) for images at distance d: below the truncation (rg / d)^(L + 1) as
  // long as rs^2 <= rg d.
  const double ax = L.d1x / P.n1, ay = L.d1y / P.n1, bx = L.d2x / P.n2, by = L.d2y / P.n2;
  const double dp = (ax + bx) * (ax + bx) + (ay + by) * (ay + by), dm = (ax - bx) * (ax - bx) + (ay - by) * (ay - by);
  const double rg = 0.5 * sqrt((dp > dm ? dp : dm) + P.hz * P.hz);
  P.rs = fmin(fmin(2.0 * rg, sqrt(rg * S.dblk)), fmax(2.0 / L.k, rg));
}
// Coefficients that a domain's table should have room for (48 bytes each with the samples), from what the host
// knows before the elements are looked at: plans for `npairs` evaluations by `ne` elements on a surface of about the
// cell's size, as tall as the cell is wide or (zlen > 0) zlen.  Half as much again as the cheapest (90 seeded
// spheres and cones of 24 to 864 elements want 0.4 to 1.9 times that plan's, nine in ten up to 1.4; a domain that
// wants more takes a higher degree), and 2.5 times the smallest, which has no higher degree to turn to.  At least
// SMT_CAPMIN and at most SMT_CAPMAX; 0 where the lattice has none.
#define SMT_CAPMIN (1LL << 18)  // 13 MB
#define SMT_CAPMAX (1LL << 22)  // 200 MB
inline long long smooth_capacity(const QPLattice& L, const SmoothLat& S, int ne, double npairs, double near, double zlen)
{
  if (!S.ok) return 0;
  // (elements small enough for a smooth rule: the real ones may be)
  const double w = sqrt(fabs(L.detd)), h = fmin(0.53 * w / sqrt((double)ne), 0.29 * S.dimg);
  const SmoothExt X = {h, zlen > 0.0 ? zlen : w, 1.0, 1.0, 1.42 * h, 0.2};
  double best = 1e300, want = 0.0, least = 1e300;
  for (int d = SMT_LMIN; d <= SMT_LMAX; d++) {
    SmoothGrid g;
    double c;
    smooth_choose(L, S, X, npairs, near, 0, 1LL << 40, d, g, c);
    if (!(c < 1e300)) continue;
    const double n = (double)g.ncent * smt_ncoef(d);
    least = fmin(least, n);
    if (c < best) {
      best = c;
      want = 1.5 * n;
    }
  }
  if (least < 1e300) want = fmax(want, 2.5 * least);
  return want < (double)SMT_CAPMIN ? SMT_CAPMIN : want > (double)SMT_CAPMAX ? SMT_CAPMAX : (long long)want;
}

// A table for `evals` evaluations at field points within the domain's extents X (zlen: the largest height of a point
// against an element): its coefficients (0: none holds) and its cost.
inline long long smooth_field_room(const QPLattice& L, const SmoothLat& S, const SmoothExt& X, double evals, double near,
                                   int tri, double chain, double& cost)
{
  cost = 1e300;
  double want = 0.0;
  for (int d = SMT_LMIN; d <= SMT_LMAX; d++) {
    SmoothGrid g;
    double c;
    smooth_choose(L, S, X, evals, near, tri, SMT_CAPMAX, d, g, c, chain);
    if (g.on && c < cost) {
      cost = c;
      want = (double)g.ncent * smt_ncoef(d);
    }
  }
  return want > 0.0 ? (long long)(1.125 * want) + SMT_PAD : 0;  // the device's rounding may add a row of centres
}

// sphere nodes and smooth rules
BEM_HD void smooth_tables_a(SmoothPlan& P, int part, int nparts)
{
  for (int i = part; i < P.nth; i += nparts) {
    smooth_gauss(P.nth, i, P.cth[i], P.wth[i]);
    P.sth[i] = sqrt((1.0 - P.cth[i]) * (1.0 + P.cth[i]));
  }
  for (int i = part; i < P.nph; i += nparts) {
    const cplx e = expi(2.0 * QP_PI * i / P.nph);
    P.cph[i] = e.re;
    P.sph[i] = e.im;
  }
  int n = 1;
  while (n * n < P.nq4) n++;
  for (int q = part; q < P.nq4; q += nparts) {
    double a, wa, b, wb;
    smooth_gauss(n, q / n, a, wa);
    smooth_gauss(n, q % n, b, wb);
    P.q4[3 * q] = a; P.q4[3 * q + 1] = b; P.q4[3 * q + 2] = wa * wb;
  }
  n = 1;
  while (n * (n + 1) < P.nq3) n++;
  // triangle: u along the edge direction from vertex 0, v across (collapsed square), weights summing
  // to 12 as those of the 3 x 12 x 12 rule
  for (int q = part; q < P.nq3; q += nparts) {
    double a, wa, b, wb;
    smooth_gauss(n + 1, q / n, a, wa);
    smooth_gauss(n, q % n, b, wb);
    const double u = 0.5 * (1.0 + a), v = 0.5 * (1.0 + b);
    // V0 = (-1/2, -s), V1 = (1, 0), V2 = (-1/2, s), s = sqrt(3) / 2
    P.q3[3 * q] = -0.5 + 1.5 * u - 1.5 * u * v;
    P.q3[3 * q + 1] = EL_SQ3 * (-0.5 + 0.5 * u + 0.5 * u * v);
    P.q3[3 * q + 2] = 6.0 * wa * wb * u;
  }
}
// projection weights: w_t p_lm(theta_t) / (norm rs^l f_l(rs)) x (1 or 2) / nph.  Stage b fills
// p_lm(theta_t), stage c scales each (m, l).
BEM_HD void smooth_tables_b(SmoothPlan& P, int part, int nparts)
{
  for (int i = part; i < (P.L + 1) * P.nth; i += nparts) {
    const int m = i / P.nth, t = i - m * P.nth;
    double a = 1.0, b = 0.0;
    for (int q = 0; q < m; q++) a *= P.sth[t];
    for (int l = m; l <= P.L; l++) {
      P.proj[smt_lm(P.L, m, l) * P.nth + t] = a;
      const double n = P.cth[t] * a - smt_rec.c[m][l + 1] * b;
      b = a;
      a = n;
    }
  }
}
BEM_HD void smooth_tables_c(SmoothPlan& P, double k, int part, int nparts)
{
  double rad[SMT_LMAX + 2];
  smooth_radial(k, P.rs * P.rs, P.L, P.top, rad, 1);
  if (part == 0) P.c00 = 1.0 / rad[0];
  for (int i = part; i < (P.L + 1) * (P.L + 1); i += nparts) {
    const int m = i / (P.L + 1), l = i - m * (P.L + 1);
    if (l < m) continue;
    double* w = P.proj + smt_lm(P.L, m, l) * P.nth;
    double nn = 0.0, rl = 1.0;
    for (int t = 0; t < P.nth; t++) nn += P.wth[t] * w[t] * w[t];
    for (int q = 0; q < l; q++) rl *= P.rs;
    const double f = (m ? 2.0 : 1.0) / (P.nph * nn * rl * rad[l]);
    for (int t = 0; t < P.nth; t++) w[t] *= P.wth[t] * f;
  }
}

// The element's contribution to the extents.
BEM_HD void smooth_extent(const QPLattice& L, const Elem& e, double* half_edge, double* radius, double* bend, double* lo,
                          double* hi)
{
  double w0 = 0.0, w1 = 0.0, w2 = 0.0;
  for (int i = 0; i < 3; i++) {
    w0 += e.cw[i][0] * e.cw[i][0];
    w1 += e.cw[i][1] * e.cw[i][1];
    w2 += e.cw[i][2] * e.cw[i][2];
  }
  *bend = fmax(*bend, sqrt((w1 > w2 ? w1 : w2) / w0));
  double v[4][3];
  const int nv = e.nn;
  const double zq[4] = {-1.0, 1.0, 1.0, -1.0}, eq[4] = {-1.0, -1.0, 1.0, 1.0};
  const double zt[3] = {-0.5, 1.0, -0.5}, et[3] = {-0.5 * EL_SQ3, 0.0, 0.5 * EL_SQ3};
  for (int j = 0; j < nv; j++) {
    const double z = (nv == 4) ? zq[j] : zt[j], n = (nv == 4) ? eq[j] : et[j];
    double r2 = 0.0;
    for (int i = 0; i < 3; i++) {
      v[j][i] = e.cr[i][0] + e.cr[i][1] * z + e.cr[i][2] * n + e.cr[i][3] * z * n;
      const double d = v[j][i] - e.cr[i][0];
      r2 += d * d;
    }
    *radius = fmax(*radius, sqrt(r2));
    const double u = (v[j][0] * L.d2y - v[j][1] * L.d2x) * L.idd, w = (v[j][1] * L.d1x - v[j][0] * L.d1y) * L.idd;
    const double p[3] = {u, w, v[j][2]};
    for (int i = 0; i < 3; i++) { lo[i] = fmin(lo[i], p[i]); hi[i] = fmax(hi[i], p[i]); }
  }
  for (int j = 0; j < nv; j++) {
    const int n = (j + 1 == nv) ? 0 : j + 1;
    double d2 = 0.0;
    for (int i = 0; i < 3; i++) d2 += (v[n][i] - v[j][i]) * (v[n][i] - v[j][i]);
    *half_edge = fmax(*half_edge, 0.5 * sqrt(d2));
  }
}

// Lattice shift that brings v (element centre minus node) into the cell around the origin, and the
// Bloch phase of it; 1 when there is a shift.
BEM_HD int smooth_shift(const QPLattice& L, const double* v, double* sx, double* sy)
{
  const double l1 = floor((v[0] * L.d2y - v[1] * L.d2x) * L.idd + 0.5);
  const double l2 = floor(-(v[0] * L.d1y - v[1] * L.d1x) * L.idd + 0.5);
  *sx = -(l1 * L.d1x + l2 * L.d2x);
  *sy = -(l1 * L.d1y + l2 * L.d2y);
  return l1 != 0.0 || l2 != 0.0;
}

// 1 when element e lies in the plane of the node at height z.
BEM_HD int smooth_in_plane(const QPLattice& L, const Elem& e, double z)
{
  const double d = fabs(e.cr[2][0] - z) + fabs(e.cr[2][1]) + fabs(e.cr[2][2]) + fabs(e.cr[2][3]);
  return d * d < SMT_ZPLANE * SMT_ZPLANE * fabs(L.detd);
}

// One smooth point of a pair added to its sums (unscaled, as accp_point's); rt the node, (sx, sy) the
// pair's shift.
BEM_HD void smooth_point(const Elem& e, const QPLattice& L, const SmoothPlan& P, const cplx* __restrict__ tab,
                         const double* rt, double sx, double sy, int q, double* rad, int st, cplx& gw, cplx& hw, double& zeta,
                         double& eta)
{
  const double* t = (e.nn == 4) ? P.q4 : P.q3;
  zeta = t[3 * q];
  eta = t[3 * q + 1];
  const double w = t[3 * q + 2];
  double r[3], W[3];
  point_geom(e, zeta, eta, rt, r, W);
  r[0] += sx;
  r[1] += sy;
  cplx g, h;
  smooth_rest(L, P, tab, r, W, rad, st, g, h);
  gw = g * ((e.nn == 4) ? w * vnorm3(W) : w);
  hw = h * w;
}

// One rule point of the nearest image, with the solid-angle terms: accp_point with g0(r) for G.
BEM_HD void smooth_near(const Elem& e, double k, const double* rt, const double* v0, const double* v1, double sx, double sy,
                        int shifted, double zeta, double eta, double w, AccP& a)
{
  double vR[3], vW[3];
  point_geom(e, zeta, eta, rt, vR, vW);
  const double R2 = dot3(vR, vR);
  const double i_aR = rsqrt_(R2), i2 = i_aR * i_aR;
  const double RW = dot3(vR, vW);
  double gi = i_aR, gR2 = R2, gRW = RW;
  if (shifted) {
    const double x = vR[0] + sx, y = vR[1] + sy;
    gR2 = x * x + y * y + vR[2] * vR[2];
    gi = rsqrt_(gR2);
    gRW = x * vW[0] + y * vW[1] + vR[2] * vW[2];
  }
  const double kr = k * gR2 * gi;
  const cplx g = expi(kr) * gi;
  double N[4];
  double wG = w;
  if (e.nn == 4) {
    bil_N4(zeta, eta, N);
    wG *= vnorm3(vW);
  } else {
    lit_N3(zeta, eta, N);
    N[3] = 0.0;
  }
  const cplx gw = g * wG, hw = (g * mk(-1.0, kr)) * (w * gRW * gi * gi);
  for (int i = 0; i < 4; i++) { a.G[i] += gw * N[i]; a.H[i] += hw * N[i]; }
  const double w3 = w * i2 * i_aR;
  const double t = 3.0 * RW * i2;
  a.F += w3 * RW;
  a.dF0 += w3 * (t * dot3(vR, v0) - dot3(vW, v0));
  a.dF1 += w3 * (t * dot3(vR, v1) - dot3(vW, v1));
}
