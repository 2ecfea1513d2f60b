// self.cuh -- self-element (t == s) coefficients, host+device.
//
// Each routine sums the points q = lane, lane + nlanes, ... of one quadrature piece into a flat
// accumulator, so a CUDA block (lane = threadIdx.x) and a serial host check (lane 0 of 1) run the
// same code; the kernels reduce the partial sums across the block and call the *_combine step.
//
// Periodic (open) domain -- q0_bil_dcoef_bd_vt2_cc_DV (q0_bil_dcoef_v2_cc.c:292-301) and
// q0_lit_dcoef_bd_vt2_cc_DV (q0_lit_dcoef_v2_cc.c:331-342): polar rule of q0_bil_coef_bd
// (q0_bil_coef.c:246-338) / q0_lit_coef_bd (q0_lit_coef.c:297-371) with one Green's function
// evaluation per point shared by all shape functions, plus the free-space solid angle F and
// its central-difference tangential derivatives (q0_bil_dcoef_v2_cc.c:336-454).
//
// Interior domains -- principal-value method: bil_dcoef_bd_vt2_PV (bil_dcoef_v2.c:334-339) =
// bil_coef_bd (bil_coef.c:244-342) + bil_dcoef_bd_tz0_PV / te0_PV (bil_dcoef.c:369-740, integrands
// :916-1630); lit_dcoef_bd_vt2_PV (lit_dcoef_v2.c:366-371) = lit_coef_bd (lit_coef.c:290-348) +
// lit_dcoef_bd_tz0_PV / te0_PV (lit_dcoef.c:461-638, integrands :858-952).  Pieces:
//   1 polar G (and H, F of curved quads)        2 far part D̄ε, r in [DEPS, rm] (64 nodes)
//   3 near disc Dε, r in [0, DEPS]              4 principal-value correction, theta in [0, pi]
#pragma once

#include "elem.cuh"

BEM_HD void acc_put(double* v, int i, cplx z) { v[2 * i] += z.re; v[2 * i + 1] += z.im; }
BEM_HD cplx acc_get(const double* v, int i) { return mk(v[2 * i], v[2 * i + 1]); }

struct SelfInfo {
  Elem e;
  cplx k;
  double zt, et;
  PolarSet P;
  int bil, curved;
  double Tz[3], Te[3];  // unnormalised tangents at the node
};

// Self integral around the point (zt, et) of element aid (collocation nodes use their own
// parameters; the boundary field of the force evaluation uses other points of the element).
BEM_HD void self_setup_at(const double* geo, int aid, double zt, double et, cplx k, SelfInfo& S)
{
  load_elem(geo, aid, S.e);
  S.k = k;
  S.zt = zt;
  S.et = et;
  polar_setup(S.e.nn, S.zt, S.et, S.P);
  S.bil = (S.e.nn == 4);
  S.curved = S.bil ? !bil_is_plane(S.e) : 0;
  for (int i = 0; i < 3; i++) {
    S.Tz[i] = S.e.cr[i][1] + S.e.cr[i][3] * S.et;
    S.Te[i] = S.e.cr[i][2] + S.e.cr[i][3] * S.zt;
  }
}

BEM_HD void self_setup(const double* geo, int aid, int tn, cplx k, SelfInfo& S)
{
  load_elem(geo, aid, S.e);
  S.k = k;
  S.zt = node_zeta(S.e.nn, tn);
  S.et = node_eta(S.e.nn, tn);
  polar_setup(S.e.nn, S.zt, S.et, S.P);
  S.bil = (S.e.nn == 4);
  S.curved = S.bil ? !bil_is_plane(S.e) : 0;
  for (int i = 0; i < 3; i++) {
    S.Tz[i] = S.e.cr[i][1] + S.e.cr[i][3] * S.et;
    S.Te[i] = S.e.cr[i][2] + S.e.cr[i][3] * S.zt;
  }
}

BEM_HD void self_K(const SelfInfo& S, double r, double cth, double sth, double* K)
{
  if (S.bil) bil_K(S.e, S.zt, S.et, r, cth, sth, K);
  else for (int i = 0; i < 3; i++) K[i] = S.e.cr[i][1] * cth + S.e.cr[i][2] * sth;
}
BEM_HD double self_aW(const SelfInfo& S, double zeta, double eta)
{
  if (!S.bil) return 1.0;
  double W[3];
  for (int i = 0; i < 3; i++) W[i] = S.e.cw[i][0] + S.e.cw[i][1] * zeta + S.e.cw[i][2] * eta;
  return vnorm3(W);
}
BEM_HD void self_N(const SelfInfo& S, double zeta, double eta, double* N)
{
  if (S.bil) bil_N4(zeta, eta, N);
  else { lit_N3(zeta, eta, N); N[3] = 0.0; }
}

// lit_dNn_pr_cs (lit_dcoef.c:845-855)
BEM_HD double lit_dN(int n, double cth, double sth)
{
  const double i_a = 0.5 / EL_P34_N0;
  if (n == 0) return -2.0 / 3.0 * i_a * (cth + EL_SQ3 * sth);
  if (n == 1) return 4.0 / 3.0 * i_a * cth;
  return -2.0 / 3.0 * i_a * (cth - EL_SQ3 * sth);
}

#define SELF_NV 40  // accumulator length of every piece

// ---- interior pieces -------------------------------------------------------------------------
// Along a ray (fixed theta) the map's K, the normal W, the products K.T with the tangents and the shape
// functions are polynomials in r (degrees 1, 1, 1, 2):
//   K = K0 + K1 r,  W = W0 + W1 r,  K.Tz = z0 + z1 r,  K.Te = e0 + e1 r,  N_i = a_i + b_i r + c_i r^2.
// Each piece's points therefore add a few scalars to moments sum f r^m, without shape functions, and the
// moments become the shape functions' sums once per ray.  The trigonometry of theta (its sine and
// cosine, three more sines for the edge distance) is also done once per ray, not at each of its points.
struct SelfRay {
  double cth, sth, K0[3], K1[3], W0[3], W1[3], z0, z1, e0, e1;
};
BEM_HD void self_ray(const SelfInfo& S, double theta, SelfRay& Y)
{
#if defined(__CUDA_ARCH__)
  sincos(theta, &Y.sth, &Y.cth);
#else
  Y.sth = sin(theta);
  Y.cth = cos(theta);
#endif
  const Elem& e = S.e;
  for (int i = 0; i < 3; i++) {
    Y.K0[i] = e.cr[i][1] * Y.cth + e.cr[i][2] * Y.sth + e.cr[i][3] * (S.zt * Y.sth + S.et * Y.cth);
    Y.K1[i] = e.cr[i][3] * (Y.cth * Y.sth);
    Y.W0[i] = e.cw[i][0] + e.cw[i][1] * S.zt + e.cw[i][2] * S.et;
    Y.W1[i] = e.cw[i][1] * Y.cth + e.cw[i][2] * Y.sth;
  }
  Y.z0 = dot3(Y.K0, S.Tz); Y.z1 = dot3(Y.K1, S.Tz);
  Y.e0 = dot3(Y.K0, S.Te); Y.e1 = dot3(Y.K1, S.Te);
}
BEM_HD double ray_K2(const SelfRay& Y, double r)  // |K|^2
{
  const double x = Y.K0[0] + Y.K1[0] * r, y = Y.K0[1] + Y.K1[1] * r, z = Y.K0[2] + Y.K1[2] * r;
  return x * x + y * y + z * z;
}
BEM_HD double ray_aW(const SelfInfo& S, const SelfRay& Y, double r)  // |W| (1 on triangles)
{
  if (!S.bil) return 1.0;
  const double x = Y.W0[0] + Y.W1[0] * r, y = Y.W0[1] + Y.W1[1] * r, z = Y.W0[2] + Y.W1[2] * r;
  const double w2 = x * x + y * y + z * z;
  return w2 * rsqrt_(w2);
}
// N_i = n[0] + n[1] r + n[2] r^2 along the ray
BEM_HD void ray_N(const SelfInfo& S, const SelfRay& Y, int i, double* n)
{
  if (S.bil) {
    const double i_a = 1.0 / EL_P44_N;
    const double u = (i == 0 || i == 3) ? -i_a : i_a, v = (i < 2) ? -i_a : i_a;
    const double a = 1.0 + u * S.zt, b = 1.0 + v * S.et;
    n[0] = 0.25 * a * b;
    n[1] = 0.25 * (a * v * Y.sth + b * u * Y.cth);
    n[2] = 0.25 * u * v * Y.cth * Y.sth;
    return;
  }
  n[2] = 0.0;
  if (i == 3) { n[0] = n[1] = 0.0; return; }
  const double h = 0.5 / EL_P34_N0 / 3.0;
  const double u = (i == 1) ? 2.0 * h : -h, v = (i == 1) ? 0.0 : (i == 0 ? -h * EL_SQ3 : h * EL_SQ3);
  n[0] = 1.0 / 3.0 + u * S.zt + v * S.et;
  n[1] = u * Y.cth + v * Y.sth;
}
// e^{i z} of a complex z
BEM_HD cplx self_cis(cplx z)
{
  cplx u = expi(z.re);
  if (z.im != 0.0) u = u * exp(-z.im);
  return u;
}
BEM_HD void csincos_(cplx z, cplx& s, cplx& c)
{
  const cplx u = expi(z.re);
  double ch = 1.0, sh = 0.0;
  if (z.im != 0.0) { ch = cosh(z.im); sh = sinh(z.im); }
  s = mk(u.im * ch, u.re * sh);
  c = mk(u.re * ch, -u.im * sh);
}
// Moments of a ray: g (times K.T) and p (times K.T, of the curved part), q: sums f r^m
struct SelfMom {
  cplx g[4], p[4], q[3];
  double f0, f1, f2;  // w / (r |K|^5): 1, r; w / (r |K|^3)
};
BEM_HD void mom_zero(SelfMom& m)
{
  for (int i = 0; i < 4; i++) { m.g[i] = mk(0, 0); m.p[i] = mk(0, 0); }
  for (int i = 0; i < 3; i++) m.q[i] = mk(0, 0);
  m.f0 = m.f1 = m.f2 = 0.0;
}
template <int N>
BEM_HD void mom_add(cplx* m, cplx f, double r)
{
  m[0] += f;
  double t = r;
  for (int i = 1; i < N; i++) {
    m[i].re += f.re * t;
    m[i].im += f.im * t;
    t *= r;
  }
}
// Adds a ray's moments to the sums of the pieces 2-4 (layout below): dG from g, dH and dF from p, q, f.
BEM_HD void ray_add(const SelfInfo& S, const SelfRay& Y, const SelfMom& m, double* v)
{
  cplx gz[3], ge[3], hz[3], he[3];
  const double cs = Y.cth * Y.sth;
  for (int k = 0; k < 3; k++) {
    gz[k] = m.g[k] * Y.z0 + m.g[k + 1] * Y.z1;
    ge[k] = m.g[k] * Y.e0 + m.g[k + 1] * Y.e1;
    if (S.curved) {
      hz[k] = (m.p[k] * Y.z0 + m.p[k + 1] * Y.z1) * cs - m.q[k] * Y.sth;
      he[k] = (m.p[k] * Y.e0 + m.p[k + 1] * Y.e1) * cs - m.q[k] * Y.cth;
    }
  }
  for (int i = 0; i < 4; i++) {
    double n[3];
    ray_N(S, Y, i, n);
    acc_put(v, i, gz[0] * n[0] + gz[1] * n[1] + gz[2] * n[2]);
    acc_put(v, 4 + i, ge[0] * n[0] + ge[1] * n[1] + ge[2] * n[2]);
    if (S.curved) {
      acc_put(v, 8 + i, hz[0] * n[0] + hz[1] * n[1] + hz[2] * n[2]);
      acc_put(v, 12 + i, he[0] * n[0] + he[1] * n[1] + he[2] * n[2]);
    }
  }
  if (S.curved) {
    v[32] += Y.sth * (3.0 * Y.cth * (Y.z0 * m.f0 + Y.z1 * m.f1) - m.f2);
    v[33] += Y.cth * (3.0 * Y.sth * (Y.e0 * m.f0 + Y.e1 * m.f1) - m.f2);
  }
}

// piece 1 layout: G[4] 0..7, H[4] 8..15, F 16
BEM_HD void self_int_piece1(const SelfInfo& S, const double* xl, const double* wl, const double* xh, const double* wh,
                            int lane, int nlanes, double* v)
{
  const int n = S.P.nsub * 128;
#if defined(__CUDA_ARCH__)
#pragma unroll 1
#endif
  for (int tq = lane; tq < n; tq += nlanes) {
    const int j = tq >> 7, m2 = tq & 127;
    double theta, wt;
    polar_theta(S.P, j, m2, xh, wh, theta, wt);
    const double rm = polar_rm(S.P, j, theta);
    SelfRay Y;
    self_ray(S, theta, Y);
    cplx g[3] = {mk(0, 0), mk(0, 0), mk(0, 0)}, h[3] = {mk(0, 0), mk(0, 0), mk(0, 0)};
    double f = 0.0;
#if defined(__CUDA_ARCH__)
#pragma unroll 1
#endif
    for (int ir = 0; ir < 12; ir++) {
      const double r = 0.5 * rm * (xl[ir] + 1.0), w = wt * 0.5 * rm * wl[ir];
      const double K2 = ray_K2(Y, r), iK = rsqrt_(K2);
      const cplx kR = S.k * (K2 * iK * r);
      const cplx ce = self_cis(kR);
      mom_add<3>(g, ce * (w * iK * ray_aW(S, Y, r)), r);
      if (S.curved) {
        const double i3 = iK * iK * iK * w;
        mom_add<3>(h, (mk(-kR.im - 1.0, kR.re) * ce) * i3, r);  // (i kR - 1) e^{ikR} / |K|^3
        f += i3;
      }
    }
    const double cs = Y.cth * Y.sth;
    for (int i = 0; i < 4; i++) {
      double N[3];
      ray_N(S, Y, i, N);
      acc_put(v, i, g[0] * N[0] + g[1] * N[1] + g[2] * N[2]);
      if (S.curved) acc_put(v, 4 + i, (h[0] * N[0] + h[1] * N[1] + h[2] * N[2]) * cs);
    }
    if (S.curved) v[16] += f * cs;
  }
}

// Along a ray the integrands of piece 2 are r^{m-1} (m = 0..3) times e^{ikr|K|} and powers of |K|, from
// DEPS to the edge: 1/r needs the 64 points, but in ln r they are smooth.  24 points in ln r give the
// integrals to 5e-17 of their sums of sizes (extended precision; 20 points: 3e-13) where |K1| r <=
// |K0| / 4, the map being far from degenerate, and |k K0| r <= 4.  1 for such elements.  k_self_interior
// (FP64 pipe 58 % busy), 6,912 rows of quads on a B200: 4.73 -> 3.10 ms.
#define SELF_NLOG 24
BEM_HD int self_log_rule(const SelfInfo& S)
{
  const double a = dot3(S.Tz, S.Tz), b = dot3(S.Te, S.Te), c = dot3(S.Tz, S.Te);
  const double d = sqrt(0.25 * (a - b) * (a - b) + c * c), lo = 0.5 * (a + b) - d, hi = 0.5 * (a + b) + d;  // of |K0|^2
  double c3 = 0.0;
  if (S.bil)
    for (int i = 0; i < 3; i++) c3 += S.e.cr[i][3] * S.e.cr[i][3];
  const double r2 = 2.24 * 2.24;  // the farthest corner from a node, and |K1| <= |cr3| / 2
  return 0.25 * c3 * r2 <= 0.0625 * lo && (S.k.re * S.k.re + S.k.im * S.k.im) * hi * r2 <= 16.0;
}

// piece 2 (D̄ε) layout: dGz[4] 0..7, dGe[4] 8..15, dHz[4] 16..23, dHe[4] 24..31, dFz 32, dFe 33.
// Items: a ray, or one half of its points.  xs, ws: the 24-point rule (nullptr: always 64 points).
BEM_HD void self_int_piece2(const SelfInfo& S, const double* xh, const double* wh, int lane, int nlanes, double* v,
                            const double* xs = nullptr, const double* ws = nullptr)
{
  const bool lg = xs && self_log_rule(S);
  const int parts = (lg && S.bil) ? 1 : 2;  // on 256 threads: 512 whole rays of a quad, 768 halves of a triangle
  const int n = S.P.nsub * 128 * parts, np = (lg ? SELF_NLOG : 64) / parts;
#if defined(__CUDA_ARCH__)
#pragma unroll 1
#endif
  for (int q = lane; q < n; q += nlanes) {
    const int half = parts == 2 ? q & 1 : 0, tq = parts == 2 ? q >> 1 : q, j = tq >> 7, m2 = tq & 127;
    double theta, wt;
    polar_theta(S.P, j, m2, xh, wh, theta, wt);
    const double rm = polar_rm(S.P, j, theta);
    SelfRay Y;
    self_ray(S, theta, Y);
    SelfMom m;
    mom_zero(m);
    const double hr = lg ? 0.5 * log(rm / EL_DEPS) : 0.5 * (rm - EL_DEPS);
    const double cr = lg ? sqrt(rm * EL_DEPS) : 0.5 * (rm + EL_DEPS);
#if defined(__CUDA_ARCH__)
#pragma unroll 1
#endif
    for (int ir = np * half; ir < np * half + np; ir++) {
      double r, w;
      if (lg) {
        r = cr * exp(hr * xs[ir]);
        w = wt * hr * ws[ir] * r;
      } else {
        r = hr * xh[ir] + cr;
        w = wt * hr * wh[ir];
      }
      const double K2 = ray_K2(Y, r), iK = rsqrt_(K2), i2 = iK * iK;
      const cplx kR = S.k * (K2 * iK * r);
      const cplx cb = mk(-kR.im - 1.0, kR.re);
      const cplx ce = self_cis(kR);
      const double w3 = w * i2 * iK * recip_(r);
      const cplx qm = (cb * ce) * w3;  // (ikR - 1) e^{ikR} w / (r |K|^3)
      mom_add<4>(m.g, qm * ray_aW(S, Y, r), r);
      if (S.curved) {
        const double w5 = w3 * i2;
        mom_add<4>(m.p, ((kR * kR + 3.0 * cb) * ce) * w5, r);
        mom_add<3>(m.q, qm, r);
        m.f0 += w5;
        m.f1 += w5 * r;
        m.f2 += w3;
      }
    }
    ray_add(S, Y, m, v);
  }
}

// piece 3 (Dε) layout: dGz[4] 0..7, dGe[4] 8..15, dHz[4] 16..23, dHe[4] 24..31 (32, 33 are not used)
BEM_HD void self_int_piece3(const SelfInfo& S, const double* xl, const double* wl, const double* xh, const double* wh,
                            int lane, int nlanes, double* v)
{
  const cplx k = S.k;
  if (S.bil) {
    // theta in 4 quarter pieces of [-pi, pi] (64 nodes each), r in [0, DEPS] (12 nodes)
#if defined(__CUDA_ARCH__)
#pragma unroll 1
#endif
    for (int tq = lane; tq < 4 * 64; tq += nlanes) {
      const int piece = tq >> 6, mm = tq & 63;
      const double theta = 0.25 * QP_PI * xh[mm] + (-0.75 + 0.5 * piece) * QP_PI;
      SelfRay Y;
      self_ray(S, theta, Y);
      SelfMom m;
      mom_zero(m);
#if defined(__CUDA_ARCH__)
#pragma unroll 1
#endif
      for (int ir = 0; ir < 12; ir++) {
        const double w = 0.25 * QP_PI * wh[mm] * 0.5 * EL_DEPS * wl[ir], r = 0.5 * EL_DEPS * (xl[ir] + 1.0);
        const double K2 = ray_K2(Y, r), iK = rsqrt_(K2), i2 = iK * iK;
        const cplx kR = k * (K2 * iK * r);
        const cplx cb = mk(-kR.im - 1.0, kR.re);
        cplx cs, cc;
        csincos_(kR, cs, cc);
        const double w3 = w * i2 * iK * recip_(r);
        mom_add<4>(m.g, (cb * cs + kR * cc) * (w3 * ray_aW(S, Y, r)), r);
        if (S.curved) {
          // e^{ikR} (k kR + 3ik) / |K|^4 - i 3 sin(kR) / (r |K|^5), and e^{ikR} ik / |K|^2 - i sin(kR) / (r |K|^3)
          const cplx ce = cc + mul_i(cs), ik = mul_i(k);
          const double w5 = w3 * i2;
          mom_add<4>(m.p, (ce * (k * kR + 3.0 * ik)) * (w * i2 * i2) - mul_i(cs) * (3.0 * w5), r);
          mom_add<3>(m.q, (ce * ik) * (w * i2) - mul_i(cs) * w3, r);
        }
      }
      ray_add(S, Y, m, v);  // f0 .. f2 are zero: no solid-angle part here
    }
  } else {
    // triangle: closed form in r; theta in 4 quarter pieces (64 nodes each)
    for (int q = lane; q < 4 * 64; q += nlanes) {
      int piece = q >> 6, m = q & 63;
      double theta = 0.25 * QP_PI * xh[m] + (-0.75 + 0.5 * piece) * QP_PI;
      double w = 0.25 * QP_PI * wh[m];
      double cth = cos(theta), sth = sin(theta);
      double K[3];
      self_K(S, 0.0, cth, sth, K);
      double aK = vnorm3(K), i_aK = 1.0 / aK;
      cplx keK = k * (EL_DEPS * aK);
      cplx cc, cs;
      csincos_(keK, cs, cc);
      // (keK + i) sin + (2 - i keK) cos - 2
      cplx f = mk(keK.re, keK.im + 1.0) * cs + mk(2.0 + keK.im, -keK.re) * cc - mk(2.0, 0.0);
      double i3 = i_aK * i_aK * i_aK;
      for (int i = 0; i < 3; i++) {
        double dn = lit_dN(i, cth, sth);
        acc_put(v, i, f * (w * dn * i3 * dot3(K, S.Tz) * i_aK));
        acc_put(v, 4 + i, f * (w * dn * i3 * dot3(K, S.Te) * i_aK));
      }
    }
  }
}

// piece 4 (principal-value correction) layout as piece 2.  Items: a line through the node (the rays
// theta and theta + pi) and one half of its 12 distances.  The line at -r is the same polynomial in -r.
BEM_HD void self_int_piece4(const SelfInfo& S, const double* xl, const double* wl, const double* xh, const double* wh,
                            int lane, int nlanes, double* v)
{
  const cplx k = S.k;
  if (S.bil) {
#if defined(__CUDA_ARCH__)
#pragma unroll 1
#endif
    for (int q = lane; q < 2 * 64 * 2; q += nlanes) {
      const int half = q & 1, tq = q >> 1, piece = tq >> 6, mm = tq & 63;
      const double theta = 0.25 * QP_PI * xh[mm] + (0.25 + 0.5 * piece) * QP_PI;
      SelfRay Y;
      self_ray(S, theta, Y);
      SelfMom m;
      mom_zero(m);
#if defined(__CUDA_ARCH__)
#pragma unroll 1
#endif
      for (int ir = 12 * half; ir < 12 * half + 12; ir++) {
        // ir = 2 n (+ r_n) and 2 n + 1 (- r_n), n of the half
        const int n = ir >> 1;
        const double r0 = 0.5 * EL_DEPS * (xl[n] + 1.0), r = (ir & 1) ? -r0 : r0;
        const double w = 0.25 * QP_PI * wh[mm] * 0.5 * EL_DEPS * wl[n];
        const double K2 = ray_K2(Y, r), iK = rsqrt_(K2), i2 = iK * iK;
        cplx cs, cc;
        csincos_(k * (K2 * iK * r0), cs, cc);
        const double w3 = w * i2 * iK * recip_(r);  // the point at -r enters with the opposite sign
        mom_add<4>(m.g, cc * (w3 * ray_aW(S, Y, r)), r);
        if (S.curved) {
          const double w5 = w3 * i2;
          mom_add<4>(m.p, cc * (3.0 * w5), r);
          mom_add<3>(m.q, cc * w3, r);
          m.f0 += w5;
          m.f1 += w5 * r;
          m.f2 += w3;
        }
      }
      ray_add(S, Y, m, v);
    }
  } else {
    for (int q = lane; q < 2 * 64; q += nlanes) {
      int piece = q >> 6, m = q & 63;
      double theta = 0.25 * QP_PI * xh[m] + (0.25 + 0.5 * piece) * QP_PI;
      double w = 0.25 * QP_PI * wh[m];
      double cth = cos(theta), sth = sin(theta);
      double K[3];
      self_K(S, 0.0, cth, sth, K);
      double aK = vnorm3(K), i_aK = 1.0 / aK;
      cplx cc, cs;
      csincos_(k * (aK * EL_DEPS), cs, cc);
      double i3 = i_aK * i_aK * i_aK;
      for (int i = 0; i < 3; i++) {
        double dn = lit_dN(i, cth, sth);
        acc_put(v, i, cs * (w * dn * i3 * dot3(K, S.Tz) * i_aK));
        acc_put(v, 4 + i, cs * (w * dn * i3 * dot3(K, S.Te) * i_aK));
      }
    }
  }
}

// Combines the four pieces (R[p] = block-summed accumulator of piece p+1) with the reference's
// factors; `negative` flips H, F and their derivatives (bil_convert_CC / _dCC).
BEM_HD void self_int_combine(const SelfInfo& S, const double* R1, const double* R2, const double* R3, const double* R4,
                             int negative, cplx* CC, cplx* dCz, cplx* dCe)
{
  for (int i = 0; i < 9; i++) { CC[i] = mk(0, 0); dCz[i] = mk(0, 0); dCe[i] = mk(0, 0); }
  const double iaTz = 1.0 / vnorm3(S.Tz), iaTe = 1.0 / vnorm3(S.Te);
  const Elem& e = S.e;
  if (S.bil) {
    double bdC = e.cr[0][1] * e.cw[0][2] + e.cr[1][1] * e.cw[1][2] + e.cr[2][1] * e.cw[2][2];
    for (int i = 0; i < 4; i++) {
      CC[i] = acc_get(R1, i) * EL_I_FP;
      // dG = -I_FP/|T| (D̄ε + i Dε - PV)
      dCz[i] = (acc_get(R2, i) + mul_i(acc_get(R3, i)) - acc_get(R4, i)) * (-EL_I_FP * iaTz);
      dCe[i] = (acc_get(R2, 4 + i) + mul_i(acc_get(R3, 4 + i)) - acc_get(R4, 4 + i)) * (-EL_I_FP * iaTe);
    }
    if (S.curved) {
      for (int i = 0; i < 4; i++) {
        CC[4 + i] = acc_get(R1, 4 + i) * (EL_I_FP * bdC);
        dCz[4 + i] = (acc_get(R2, 8 + i) + acc_get(R3, 8 + i) - acc_get(R4, 8 + i)) * (bdC * EL_I_FP * iaTz);
        dCe[4 + i] = (acc_get(R2, 12 + i) + acc_get(R3, 12 + i) - acc_get(R4, 12 + i)) * (bdC * EL_I_FP * iaTe);
      }
      CC[8] = mk(R1[16] * EL_I_FP * bdC, 0);
      dCz[8] = mk((R2[32] + R4[32]) * bdC * EL_I_FP * iaTz, 0);
      dCe[8] = mk((R2[33] + R4[33]) * bdC * EL_I_FP * iaTe, 0);
    }
  } else {
    double V[3] = {e.cw[0][0], e.cw[1][0], e.cw[2][0]};
    double aW = vnorm3(V);
    cplx ik = crecip(S.k);  // 1/k
    for (int i = 0; i < 3; i++) {
      CC[i] = acc_get(R1, i) * (EL_I_SPSQ3 * aW);
      dCz[i] = (acc_get(R2, i) + mul_i(acc_get(R3, i)) * ik - acc_get(R4, i) * ik) * (-EL_I_SPSQ3 * aW * iaTz);
      dCe[i] = (acc_get(R2, 4 + i) + mul_i(acc_get(R3, 4 + i)) * ik - acc_get(R4, 4 + i) * ik) * (-EL_I_SPSQ3 * aW * iaTe);
    }
  }
  if (negative) {
    for (int i = 4; i < 9; i++) { CC[i] = -CC[i]; dCz[i] = -dCz[i]; dCe[i] = -dCe[i]; }
  }
}

// ---- periodic (open-domain) self pair ----------------------------------------------------------
// Layout: G[4] 0..7, H[4] 8..15 (polar rule with the quasi-periodic Green's function), then the
// free-space solid angle of a curved quad at the node and at its four finite-difference
// neighbours (zeta +- h, eta +- h): 16..20.  Returns the first QPGF failure code (0 if none).
// nf: how many solid-angle centres to evaluate (5 for the derivatives of the assembly, 1 when
// only F at the point is needed).
BEM_HD int self_per_points(const SelfInfo& S, const QPLattice& L, const double* xl, const double* wl, const double* xh,
                           const double* wh, int lane, int nlanes, double* v, int nf = 5)
{
  int err = 0;
  const Elem& e = S.e;
  const int npts = S.P.nsub * 128 * 12;
  for (int q = lane; q < npts; q += nlanes) {
    int ir = q % 12, tq = q / 12, j = tq >> 7, m2 = tq & 127;
    double theta, wt;
    polar_theta(S.P, j, m2, xh, wh, theta, wt);
    double rm = polar_rm(S.P, j, theta);
    double cth = cos(theta), sth = sin(theta);
    double r = 0.5 * rm * (xl[ir] + 1.0);
    double w = wt * 0.5 * rm * wl[ir];
    double zeta = r * cth + S.zt, eta = r * sth + S.et;
    double vR[3], W[3], N[4], K[3];
    self_K(S, r, cth, sth, K);
    for (int i = 0; i < 3; i++) {
      vR[i] = r * K[i];
      W[i] = S.bil ? e.cw[i][0] + e.cw[i][1] * zeta + e.cw[i][2] * eta : e.cw[i][0];
    }
    self_N(S, zeta, eta, N);
    QPVal g;
    int e2 = qpgf_eval<QP_BOTH, true>(L, vR, g);
    if (e2 < 0) err = e2;
    double aW = S.bil ? vnorm3(W) : 1.0;
    cplx gw = g.G * (w * aW * r);
    cplx hw = (g.dG[0] * W[0] + g.dG[1] * W[1] + g.dG[2] * W[2]) * (w * r);
    for (int i = 0; i < 4; i++) { acc_put(v, i, gw * N[i]); acc_put(v, 4 + i, hw * N[i]); }
  }
  if (S.bil && S.curved) {
    const double h = EL_CDFH;
    const double cz[5] = {S.zt, S.zt + h, S.zt - h, S.zt, S.zt};
    const double ce[5] = {S.et, S.et, S.et, S.et + h, S.et - h};
    for (int c = 0; c < nf; c++) v[16 + c] += bil_self_F(e, cz[c], ce[c], xl, wl, xh, wh, lane, nlanes);
  }
  return err;
}

BEM_HD void self_per_combine(const SelfInfo& S, const double* R, cplx* CC, cplx* dCz, cplx* dCe)
{
  for (int i = 0; i < 9; i++) { CC[i] = mk(0, 0); dCz[i] = mk(0, 0); dCe[i] = mk(0, 0); }
  const Elem& e = S.e;
  if (S.bil) {
    for (int i = 0; i < 4; i++) { CC[i] = acc_get(R, i); CC[i + 4] = acc_get(R, 4 + i); }
    double bdC = e.cr[0][1] * e.cw[0][2] + e.cr[1][1] * e.cw[1][2] + e.cr[2][1] * e.cw[2][2];
    double s = EL_I_FP * bdC;
    CC[8] = mk(R[16] * s, 0);
    // dF/dt by central differences (q0_bil_dcoef_bd_tz0_cc_DV :336-362, te0 :364-390)
    dCz[8] = mk(1.0 / vnorm3(S.Tz) * (R[17] * s - R[18] * s) / (2.0 * EL_CDFH), 0);
    dCe[8] = mk(1.0 / vnorm3(S.Te) * (R[19] * s - R[20] * s) / (2.0 * EL_CDFH), 0);
  } else {
    double V[3] = {e.cw[0][0], e.cw[1][0], e.cw[2][0]};
    double aV = vnorm3(V);
    for (int i = 0; i < 3; i++) {
      CC[i] = acc_get(R, i) * (2.0 / (3.0 * EL_SQ3) * aV);
      CC[i + 4] = acc_get(R, 4 + i) * (2.0 / (3.0 * EL_SQ3));
    }
  }
}
