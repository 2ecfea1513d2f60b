// ewald_warp.cuh -- one quasi-periodic Green's function by a whole warp: Ewald's sums with one split
// parameter and fixed sets of terms (SmoothLat, smooth.cuh), 32 terms at a time, for the calls that need
// few evaluations soon (fields at a point) and for the second derivatives.
//
// The per-point sums (qpgf.cuh) walk the lattice term by term and stop by the size of the last one: a
// serial chain of 100 to 600 terms, 0.3 to 1.2 ms.  Here every term above 2e-17 is summed, so a warp
// needs ~15 terms per lane and no stop rule: ~15 us.  More operations in all (~400 terms against ~200),
// so it is the slower one where there are enough points to fill the GPU one thread each.
// With (k veps)^2 <= EWW_EXPM no term exceeds e^2 times the sum (e^3 in the per-point sums).
#pragma once

#include "smooth.cuh"

#define EWW_EXPM 2.0

// G, grad G and, HESS, the second derivatives (xx, yy, zz, xy, yz, zx).
struct EwaldVal {
  cplx G, dG[3], d2[6];
};

// Adds an order with a = (ax, ay) at (x, y): F, Fz its share of G and of dG/dz without e^{i a.rho} at height
// |z| (sg the sign of z), b2 = k^2 - |a|^2, c2 the Gaussian term of F''.
template <bool HESS>
BEM_HD void ewald_add(double ax, double ay, double b2, double c2, double x, double y, double sg, cplx F, cplx Fz, EwaldVal& o)
{
  const cplx ce = expi(ax * x + ay * y);
  F = F * ce;
  Fz = Fz * (ce * sg);
  o.G += F;
  const cplx iF = mul_i(F);
  o.dG[0] += iF * ax;
  o.dG[1] += iF * ay;
  o.dG[2] += Fz;
  if (HESS) {
    const cplx iz = mul_i(Fz);
    o.d2[0] += F * (-ax * ax);
    o.d2[1] += F * (-ay * ay);
    o.d2[2] += F * -b2 - ce * c2;  // F'' = -beta^2 F - (2 / (sqrt(pi) veps)) e^{...} / (4 |cell|)
    o.d2[3] += F * (-ax * ay);
    o.d2[4] += iz * ay;
    o.d2[5] += iz * ax;
  }
}

// Propagating order q of the lattice's list.
template <bool HESS>
BEM_HD void ewald_prop(const QPLattice& L, const SmoothLat& S, const QPProp& q, double x, double y, double z, double sg,
                       EwaldVal& o)
{
  const double c = 0.25 * fabs(L.idd), t = z / (2.0 * S.ve);
  const double ef = exp(q.bn2 * S.ve * S.ve - t * t);
  const cplx ff = expi(q.bn * z);
  const cplx w = faddeeva_w_upper(q.bn * S.ve, t);
  const cplx F = mk(-(ef * w.im + ff.im), ff.re) * (2.0 * c / q.bn);
  const cplx Fz = mk(ef * w.re - ff.re, -ff.im) * (2.0 * c);
  ewald_add<HESS>(q.an0, q.an1, q.bn2, 2.0 * c * QP_INV_SQRTPI / S.ve * ef, x, y, sg, F, Fz, o);
}

// Order (q1, q2), if it is evanescent (the propagating ones come from the list).
template <bool HESS>
BEM_HD void ewald_evan(const QPLattice& L, const SmoothLat& S, int q1, int q2, double x, double y, double z, double sg,
                       EwaldVal& o)
{
  const double ax = smt_add(smt_add(-L.vkx, smt_mul(q1, L.g1x)), smt_mul(q2, L.g2x));
  const double ay = smt_add(smt_add(-L.vky, smt_mul(q1, L.g1y)), smt_mul(q2, L.g2y));
  const double b2 = smt_add(smt_add(smt_mul(L.k, L.k), -smt_mul(ax, ax)), -smt_mul(ay, ay));
  if (b2 > 0.0 || -b2 * S.ve * S.ve > SMT_CUT) return;
  const double c = 0.25 * fabs(L.idd), t = z / (2.0 * S.ve);
  const double ib = rsqrt_(-b2), bn = -b2 * ib, u = bn * S.ve;
  const double ef = exp(b2 * S.ve * S.ve - t * t);
  const double f1 = ef * qp_erfcx_poly(u + t), x2 = ef * qp_erfcx_poly(fabs(u - t));
  const double f2 = (u >= t) ? x2 : 2.0 * exp(-bn * z) - x2;
  ewald_add<HESS>(ax, ay, b2, 2.0 * c * QP_INV_SQRTPI / S.ve * ef, x, y, sg, mk((f1 + f2) * c * ib, 0.0),
                  mk((f1 - f2) * c, 0.0), o);
}

// Adds image (p, q) at r, if it is within the sums' reach.
template <bool HESS>
BEM_HD void ewald_image(const QPLattice& L, const SmoothLat& S, int p, int q, const double* r, EwaldVal& o)
{
  const double X = p * L.d1x + q * L.d2x, Y = p * L.d1y + q * L.d2y;
  const double x = r[0] + X, y = r[1] + Y, z = r[2], R2 = x * x + y * y + z * z;
  if (R2 > S.rmax * S.rmax) return;
  const double iR = rsqrt_(R2), R = R2 * iR, i2 = iR * iR, ke = L.k * S.ve, iv = 1.0 / S.ve, t = 0.5 * R * iv;
  const cplx w = faddeeva_w_upper(ke, t);
  const cplx ce = expi(L.vkx * X + L.vky * Y) * (exp(ke * ke - t * t) * EL_I_FP);
  o.G += ce * (iR * w.re);
  const double f1 = i2 * (iR * w.re - L.k * w.im + iv * QP_INV_SQRTPI);
  const cplx g = ce * -f1;
  o.dG[0] += g * x;
  o.dG[1] += g * y;
  o.dG[2] += g * z;
  if (HESS) {
    const double f2 = i2 * (2.0 * L.k * L.k * iR * w.re - iv * iv * iv * QP_INV_SQRTPI);
    const cplx h = ce * (3.0 * i2 * f1 - 0.5 * f2);
    o.d2[0] += g + h * (x * x);
    o.d2[1] += g + h * (y * y);
    o.d2[2] += g + h * (z * z);
    o.d2[3] += h * (x * y);
    o.d2[4] += h * (y * z);
    o.d2[5] += h * (z * x);
  }
}

// Terms first, first + stride, ... of all the sums at r (any point; L has its list of propagating orders), without the Bloch phase of its cell;
// (*px, *py) the lattice vector of that cell.
template <bool HESS>
BEM_HD void ewald_terms(const QPLattice& L, const SmoothLat& S, const double* r_in, int first, int stride, EwaldVal& o,
                        double* px, double* py)
{
  o.G = mk(0.0, 0.0);
  for (int i = 0; i < 3; i++) o.dG[i] = mk(0.0, 0.0);
  if (HESS)
    for (int i = 0; i < 6; i++) o.d2[i] = mk(0.0, 0.0);
  const double l1 = floor((r_in[0] * L.d2y - r_in[1] * L.d2x) * L.idd + 0.5);
  const double l2 = floor(-(r_in[0] * L.d1y - r_in[1] * L.d1x) * L.idd + 0.5);
  *px = l1 * L.d1x + l2 * L.d2x;
  *py = l1 * L.d1y + l2 * L.d2y;
  const double r[3] = {r_in[0] - *px, r_in[1] - *py, r_in[2]};
  const double sg = (r[2] < 0.0) ? -1.0 : 1.0;
  const int no = S.no1 * S.no2, ni = (2 * S.m1 + 1) * (2 * S.m2 + 1);
  for (int i = first; i < L.nprop; i += stride) ewald_prop<HESS>(L, S, L.prop[i], r[0], r[1], sg * r[2], sg, o);
  for (int i = first; i < no; i += stride)
    ewald_evan<HESS>(L, S, S.o1 + i / S.no2, S.o2 + i % S.no2, r[0], r[1], sg * r[2], sg, o);
  for (int i = first; i < ni; i += stride)
    ewald_image<HESS>(L, S, i / (2 * S.m2 + 1) - S.m1, i % (2 * S.m2 + 1) - S.m2, r, o);
}

// Applies the cell's Bloch phase.
template <bool HESS>
BEM_HD void ewald_phase(const QPLattice& L, double px, double py, EwaldVal& o)
{
  if (px == 0.0 && py == 0.0) return;
  const cplx f = expi(-(L.vkx * px + L.vky * py));
  o.G = o.G * f;
  for (int i = 0; i < 3; i++) o.dG[i] = o.dG[i] * f;
  if (HESS)
    for (int i = 0; i < 6; i++) o.d2[i] = o.d2[i] * f;
}
