"""The tabulated smooth remainder of the assembly's Green's function (csrc/smooth.cuh), pair by pair on
the host build, against an Ewald sum with a small split parameter (numpy, scipy's w and erfcx) and
against the plain lattice sums of the same build.

Tolerance: the expansions and the smooth rules are truncated below 5e-16 (SMT_TOL, SMT_QTOL), rounding
adds a few 1e-15 of the parts' size, so G and H of a pair must agree with the reference to 1e-13 of its
largest entry of each kind plus 1e-14 of the size the cancelling parts have (the pair's near and smooth
parts, at most a few times the largest G times 1 / distance).  The plain sums' own error grows with the
wave number (their terms reach e^3 times the sum, which itself may be small): they must agree to ten times
that.  F and its derivatives come from the same points and differ by rounding only (1e-13 of the
largest)."""
import ctypes as C
import math
import os
import subprocess

import numpy as np
import pytest

from conftest import BUILD, REPO


@pytest.fixture(scope="module")
def sh():
    os.makedirs(BUILD, exist_ok=True)
    so = os.path.join(BUILD, "libsmooth_host.so")
    src = os.path.join(REPO, "tests", "native", "smooth_host.cpp")
    hdr = os.path.join(REPO, "bem3_emf_qd2_b200", "csrc")
    newest = max(os.path.getmtime(os.path.join(hdr, f)) for f in os.listdir(hdr))
    if not os.path.exists(so) or os.path.getmtime(so) < max(newest, os.path.getmtime(src)):
        subprocess.run(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-x", "c++", "-I" + hdr, src, "-o", so], check=True)
    lib = C.CDLL(so)
    vp, i, d = C.c_void_p, C.c_int, C.c_double
    lib.sh_plan.argtypes = [vp, vp, i, d, i, vp]
    lib.sh_pair.argtypes = [vp, i, i, i, i, i, vp, vp, vp, vp]
    lib.sh_ewald.argtypes = [vp, vp, i, i, vp, vp]
    lib.sh_rule.argtypes = [vp, i, vp, vp, vp, d, d, i, vp, vp]
    lib.sh_self2.argtypes = [vp, i, i, d, d, vp, vp, vp, vp, vp, vp]
    return lib


def _elements(rng, tri, half, z0):
    """Geometry records (slot 0 unused) of 6 elements of half edge ~ `half`, spread over +-0.7 in the
    plane and +-z0 in height, oriented at random, bilinear quads slightly twisted."""
    from bem3_emf_qd2_b200.dqd2 import ET34, ET44, ZT34, ZT44, element_constants
    n = 6
    rn, ed = [np.zeros(3)], [[0, 0, 0, 0]]
    for _ in range(n):
        c = np.array([rng.uniform(-0.7, 0.7), rng.uniform(-0.7, 0.7), rng.uniform(-z0, z0)])
        q, _ = np.linalg.qr(rng.normal(size=(3, 3)))
        shape = [(-1, -1), (1, -1), (1, 1), (-1, 1)] if not tri else [(-1, -0.8), (1, -0.9), (0.1, 1)]
        ids = []
        for a, b in shape:
            p = np.array([a * half, b * half * 0.9, 0.08 * half * a * b])
            rn.append(c + q @ p)
            ids.append(len(rn) - 1)
        ed.append(ids + [0] * (4 - len(ids)))
    rn, ed = np.array(rn), np.array(ed, np.int32)
    cr, cw = element_constants(rn, ed)
    geo = np.zeros((n + 1, 48))
    for e in range(1, n + 1):
        geo[e, 0:12], geo[e, 12:21] = cr[e].ravel(), cw[e].ravel()
        for j in range(4):
            z, t = (ZT34[j], ET34[j]) if tri else (ZT44[j], ET44[j])
            geo[e, 21 + 3 * j:24 + 3 * j] = cr[e, :, 0] + cr[e, :, 1] * z + cr[e, :, 2] * t + cr[e, :, 3] * z * t
        geo[e, 45] = 3 if tri else 4
    return np.ascontiguousarray(geo)


def _green(lat, r):
    """G and grad G [n, 4] by Ewald's method with (k ve)^2 <= 1/2, all terms above 1e-18."""
    from scipy.special import erfcx, wofz
    k, kx, ky = lat[:3]
    d1, d2 = lat[3:5], lat[5:7]
    det = d1[0] * d2[1] - d2[0] * d1[1]
    l1 = np.floor((r[:, 0] * d2[1] - r[:, 1] * d2[0]) / det + 0.5)
    l2 = np.floor(-(r[:, 0] * d1[1] - r[:, 1] * d1[0]) / det + 0.5)
    R = l1[:, None] * d1 + l2[:, None] * d2
    x, y, z = r[:, 0] - R[:, 0], r[:, 1] - R[:, 1], r[:, 2]
    n1, n2, A = np.linalg.norm(d1), np.linalg.norm(d2), abs(det)
    ve = min(math.sqrt(A / (4 * math.pi)), math.sqrt(0.5) / k)
    ke = k * ve
    out = np.zeros((len(x), 4), complex)
    reach = 2 * ve * math.sqrt(42 + ke * ke) + 0.5 * (n1 + n2)
    m1, m2 = int(reach * n2 / A) + 2, int(reach * n1 / A) + 2
    for a in range(-m1, m1 + 1):
        for b in range(-m2, m2 + 1):
            px, py = x + a * d1[0] + b * d2[0], y + a * d1[1] + b * d2[1]
            D = np.sqrt(px * px + py * py + z * z)
            if D.min() > reach:
                continue
            q = D / (2 * ve)
            ef, w = np.exp(ke * ke - q * q), wofz(ke + 1j * q)
            cb = np.exp(1j * (kx * (a * d1[0] + b * d2[0]) + ky * (a * d1[1] + b * d2[1]))) / (4 * math.pi)
            cf = -cb * ef * (w.real / D - k * w.imag + 1 / (ve * math.sqrt(math.pi))) / (D * D)
            out += np.stack([cb * ef * w.real / D, cf * px, cf * py, cf * z], -1)
    # the reciprocal vectors as the library rounds them: near a grazing order (k = |a|) the sum depends on
    # their last bits
    idd = 1.0 / det
    g1 = np.array([2 * math.pi * idd * d2[1], -2 * math.pi * idd * d2[0]])
    g2 = np.array([-2 * math.pi * idd * d1[1], 2 * math.pi * idd * d1[0]])
    amax = math.sqrt(42 / ve ** 2 + k * k) + math.hypot(kx, ky)
    az, sz, q = np.abs(z), np.where(z < 0, -1.0, 1.0), np.abs(z) / (2 * ve)
    for a in range(-int(amax * n1 / 6.28) - 2, int(amax * n1 / 6.28) + 3):
        for b in range(-int(amax * n2 / 6.28) - 2, int(amax * n2 / 6.28) + 3):
            ax, ay = -kx + a * g1[0] + b * g2[0], -ky + a * g1[1] + b * g2[1]
            b2 = k * k - ax * ax - ay * ay
            if -b2 * ve * ve > 42:
                continue
            bn, ce = math.sqrt(abs(b2)), np.exp(1j * (ax * x + ay * y))
            ef, u = np.exp(b2 * ve * ve - q * q), bn * ve
            if b2 > 0:
                w, ff = wofz(u + 1j * q), np.exp(1j * bn * az)
                F, dz = ce * (2 / bn) * (ff + 1j * ef * w.imag), 2 * ce * (ef * w.real - ff) * sz
            else:
                f1 = ef * erfcx(u + q)
                f2 = np.where(q <= u, ef * erfcx(np.maximum(u - q, 0)), 2 * np.exp(-bn * az) - ef * erfcx(np.maximum(q - u, 0)))
                F, dz = -1j * ce * (f1 + f2) / bn, ce * (f1 - f2) * sz
            out += 0.25 / A * np.stack([1j * F, -ax * F, -ay * F, dz], -1)
    return out * np.exp(-1j * (kx * R[:, 0] + ky * R[:, 1]))[:, None]


def _reference(lat, geo, t, tn, s):
    """G[4], H[4] of the pair by the 12 x 12 rule (3 x 12 x 12 on triangles), scaled as the matrices are."""
    x, w = np.polynomial.legendre.leggauss(12)
    a, b, ww = np.repeat(x, 12), np.tile(x, 12), np.repeat(w, 12) * np.tile(w, 12)
    cr, cw, q3 = geo[s, :12].reshape(3, 4), geo[s, 12:21].reshape(3, 3), math.sqrt(3)
    if geo[s, 45] == 4:
        z, e, wq, aux = a, b, ww, 1 / math.sqrt(3)
        N = np.stack([(1 - z / aux) * (1 - e / aux), (1 + z / aux) * (1 - e / aux), (1 + z / aux) * (1 + e / aux),
                      (1 - z / aux) * (1 + e / aux)], -1) / 4
        W = cw[:, 0] + np.outer(z, cw[:, 1]) + np.outer(e, cw[:, 2])
        sg, sh = np.linalg.norm(W, axis=1), 1.0
    else:
        z = np.concatenate([(3 + 2 * a + 2 * b + a * b) / 8, (-3 + a - 5 * b - a * b) / 16, (-3 - 5 * a + b - a * b) / 16])
        e = q3 * np.concatenate([(b - a) / 8, (3 + 3 * a + b + a * b) / 16, (-3 - a - 3 * b - a * b) / 16])
        wq = np.tile(ww * (1 + a / 4 + b / 4), 3)
        N = np.stack([(1 - 2.5 * (z + q3 * e)) / 3, (1 + 5 * z) / 3, (1 - 2.5 * (z - q3 * e)) / 3, 0 * z], -1)
        W = np.tile(cw[:, 0], (len(z), 1))
        cr = cr * np.array([1, 1, 1, 0])
        sg, sh = np.linalg.norm(W, axis=1) / 24, 1 / 24
    r = cr[:, 0] + np.outer(z, cr[:, 1]) + np.outer(e, cr[:, 2]) + np.outer(z * e, cr[:, 3])
    g = _green(lat, r - geo[t, 21 + 3 * tn:24 + 3 * tn])
    return (wq * sg * g[:, 0]) @ N, (wq * sh * (g[:, 1:] * W).sum(1)) @ N


LATTICES = {
    "square": (1.0, 0.0, 0.0, 1.0), "rectangular": (0.8, 0.0, 0.0, 1.5), "hexagonal": (0.9, 0.0, 0.45, 0.7794),
    "oblique": (1.0, 0.1, 0.3, 0.9), "left_handed": (0.0, 1.1, 1.0, 0.0), "second_long": (0.9, 0.0, -0.35, 1.3),
}


def _plan(sh, rng, lattice, lam, tri, half, degree, z0=0.6):
    k = 2 * math.pi * 1.33 / lam
    th, ph = rng.uniform(0.05, 1.0), rng.uniform(0, 2 * math.pi)
    lat = np.array([k, k * math.sin(th) * math.cos(ph), k * math.sin(th) * math.sin(ph), *LATTICES[lattice]])
    geo = _elements(rng, tri, half, z0)
    info = np.zeros(5, np.int32)
    got = sh.sh_plan(lat.ctypes.data, geo.ctypes.data, 6, 1e7, degree, info.ctypes.data)
    return geo, got, info, lat


def _pair(sh, geo, t, tn, s, plain):
    from bem3_emf_qd2_b200 import gauss_legendre
    x, w = gauss_legendre(12)
    out, ip = np.zeros(19), C.c_int()
    st = sh.sh_pair(geo.ctypes.data, t, tn, s, plain, 12, x.ctypes.data, w.ctypes.data, out.ctypes.data, C.byref(ip))
    assert st >= 0
    return out[0:8:2] + 1j * out[1:8:2], out[8:16:2] + 1j * out[9:16:2], out[16:], ip.value


@pytest.mark.parametrize("lattice", sorted(LATTICES))
@pytest.mark.parametrize("tri,lam,half,degree", [
    (False, 0.532, 0.02, 0), (True, 0.7, 0.03, 0), (False, 0.8, 0.06, 0), (False, 0.4, 0.015, 0),
    (False, 0.6, 0.01, 8), (True, 0.6, 0.01, 11), (False, 0.45, 0.04, 14), (True, 0.5, 0.05, 17), (False, 0.7, 0.08, 18)])
def test_tabulated_pairs_equal_plain_lattice_sums(sh, lattice, tri, lam, half, degree):
    rng = np.random.default_rng(sum(map(ord, lattice)) * 1000 + int(lam * 1000) + degree)
    geo, got, info, lat = _plan(sh, rng, lattice, lam, tri, half, degree)
    assert got == 1
    assert degree == 0 or info[1] == degree
    for t, tn, s in ((1, 0, 2), (3, 2, 4), (5, 1, 6), (2, 2 if tri else 3, 1)):
        G, H, F, ip = _pair(sh, geo, t, tn, s, 0)
        Gp, Hp, Fp, _ = _pair(sh, geo, t, tn, s, 1)
        Gr, Hr = _reference(lat, geo, t, tn, s)
        assert ip == 0
        area = half * half * 4
        dist = np.linalg.norm(geo[s, [0, 4, 8]] - geo[t, 21 + 3 * tn:24 + 3 * tn])
        size = np.abs(Gr).max() + area / (4 * math.pi)
        tol_g = 1e-13 * np.abs(Gr).max() + 1e-14 * size
        tol_h = 1e-13 * np.abs(Hr).max() + 1e-14 * size * (10 + 1 / min(dist, 1.0))
        assert np.abs(G - Gr).max() <= tol_g, (t, s)
        assert np.abs(H - Hr).max() <= tol_h, (t, s)
        assert np.abs(G - Gp).max() <= 10 * tol_g, (t, s)
        assert np.abs(H - Hp).max() <= 10 * tol_h, (t, s)
        assert np.abs(F - Fp).max() <= 1e-13 * np.abs(Fp).max(), (t, s)


@pytest.mark.parametrize("lam,half,degree", [(0.5, 0.4, 0), (0.6, 0.02, 18), (0.25, 0.02, 0)])
def test_plan_refuses_what_it_cannot_hold(sh, lam, half, degree):
    """Elements too large for a smooth rule of 12 points have no plan; a plan that exists keeps its balls
    below the first zero of the spherical Bessel functions."""
    rng = np.random.default_rng(5)
    geo, got, info, lat = _plan(sh, rng, "square", lam, False, half, degree)
    if half > 0.3:
        assert got == 0
    else:
        assert got == 1 and info[2] > 0


def test_in_plane_pairs_are_left_to_the_lattice_sums(sh):
    """A flat element at the node's height (within 1e-11 periods) is flagged, one 1e-9 above it is not."""
    rng = np.random.default_rng(9)
    geo, got, _, _ = _plan(sh, rng, "square", 0.6, True, 0.03, 12)
    assert got == 1
    for dz, want in ((0.0, 1), (5e-17, 1), (1e-9, 0), (0.01, 0)):
        g = geo.copy()
        g[2, 8:12] = [g[1, 23] + dz, 0.0, 0.0, 0.0]  # z of element 2's map: constant
        ip = C.c_int()
        out, x = np.zeros(19), np.zeros(1)
        sh.sh_pair(g.ctypes.data, 1, 0, 2, 0, 0, x.ctypes.data, x.ctypes.data, out.ctypes.data, C.byref(ip))
        assert ip.value == want, dz


@pytest.mark.parametrize("lattice", sorted(LATTICES))
@pytest.mark.parametrize("lam", [0.4, 0.8, 2.5])
def test_warp_sums_equal_the_reference_and_the_plain_second_derivatives(sh, lattice, lam):
    """ewald_warp.cuh: G and grad G against the numpy sums, the second derivatives against qpgf_eval2, at
    points of every height (0 and far among them) and in other cells.  Rounding: terms up to e^2 (the
    plain sums e^3) times the sum, ~400 of them: 1e-13 and, for the plain sums at large wave numbers, 1e-11
    of the largest value."""
    rng = np.random.default_rng(int(lam * 100))
    k = 2 * math.pi * 1.33 / lam
    lat = np.array([k, 0.3 * k, -0.2 * k, *LATTICES[lattice]])
    n = 12
    r = np.concatenate([rng.uniform(-1.6, 1.6, (n, 2)), rng.uniform(-0.9, 0.9, (n, 1))], 1)
    r[:4, 2] = [0.0, 1e-9, -2.5, 1.3]
    r = np.ascontiguousarray(r)
    out, plain = np.zeros((n, 20)), np.zeros((n, 20))
    assert sh.sh_ewald(lat.ctypes.data, r.ctypes.data, n, 32, out.ctypes.data, plain.ctypes.data) == 1
    out, plain, ref = out.view(complex), plain.view(complex), _green(lat, r)
    assert np.max(np.abs(out[:, :4] - ref) / np.abs(ref).max(1, keepdims=True)) <= 1e-13
    assert np.max(np.abs(out - plain) / np.abs(plain).max(1, keepdims=True)) <= 1e-11


# rule_order's limits: distance over the half edge, wave number times it
RULES = {6: (33.0, 0.25), 7: (17.0, 0.55), 8: (10.5, 0.95), 9: (7.4, 1.45), 10: (5.6, 2.0), 11: (4.6, 2.7)}


@pytest.mark.parametrize("tri", [False, True])
@pytest.mark.parametrize("n", sorted(RULES))
def test_fewer_points_for_distant_pairs(sh, tri, n):
    """The n-point rule just inside its limits of distance and wave number, against 30 points, the
    integrands in extended precision.  Tolerance: 2e-16 of the integrand's size for each of the two
    directions, tripled for the shape functions (up to 1.4 a direction); just outside, more points are
    taken."""
    rng = np.random.default_rng(100 * n + tri)
    q, kh = RULES[n]
    s3 = math.sqrt(3)
    for trial in range(24):
        half = 10.0 ** rng.uniform(-2, -1)
        geo = _elements(rng, tri, half, 0.6)
        s = 1 + trial % 6
        cr = geo[s, :12].reshape(3, 4)
        if tri:
            p, t = 0.375 * cr[:, 1], 0.125 * s3 * cr[:, 2]
            h, off = math.sqrt(max(p @ p + t @ t + 2 * abs(p @ t), 4 * t @ t)), 2.0
        else:
            a, b, c = cr[:, 1], cr[:, 2], cr[:, 3]
            h, off = math.sqrt(c @ c + max(a @ a + 2 * abs(a @ c), b @ b + 2 * abs(b @ c))), 1.0
        part = rng.choice([0.0, 0.1, 1.0])  # of the imaginary part in the wave number's limit
        k = rng.choice([0.05, 0.5, 0.999]) * kh / h
        kre, kim = (1 - part) * k, part * k / 2.5
        u = rng.normal(size=3)
        if trial % 3 == 0:  # in line with an edge
            u = cr[:, 1 + trial // 3 % 2]
        u = u / np.linalg.norm(u)
        v0, v1 = rng.normal(size=(2, 3))
        v0, v1 = v0 / np.linalg.norm(v0), v1 / np.linalg.norm(v1)

        def run(m, dist):
            rt = np.ascontiguousarray(cr[:, 0] - u * dist)
            out, size = np.zeros(51), np.zeros(3)
            got = sh.sh_rule(geo.ctypes.data, s, rt.ctypes.data, v0.ctypes.data, v1.ctypes.data, kre, kim, m,
                             out.ctypes.data, size.ctypes.data)
            return got, out, size

        dist = (q + off) * h * 1.0001
        got, out, size = run(n, dist)
        assert got == n, (trial, got)
        _, ref, _ = run(30, dist)
        scale = np.concatenate([np.repeat(size[[0, 1, 1, 2, 1, 2]], 8), [size[1], size[2], size[2]]])
        # the solid angle is not damped
        scale[48:] *= math.exp(kim * (dist + 2 * h))
        assert (np.abs(out - ref) <= 1.2e-15 * scale).all(), (trial, (np.abs(out - ref) / scale).max())
        assert run(n, (q + off) * h * 0.9999)[0] == n + 1
        assert run(n, 1.0)[0] >= n or dist < 1.0


@pytest.mark.parametrize("shape", ["quad", "twisted", "trapezoid", "triangle"])
@pytest.mark.parametrize("kr", [0.01, 1.0, 3.95, 4.05])
def test_self_rays_in_the_logarithm(sh, shape, kr):
    """The 24-point rule in ln r against the 64-point rule in r, up to the limits of |k K| r and of the
    distortion.  Tolerance: the rules agree to 5e-17 of the sums of sizes; the rounding of 64 values (a few
    units each) per ray and the cancellation of opposite rays are covered by 2e-14 of the largest sum."""
    from bem3_emf_qd2_b200 import gauss_legendre
    from bem3_emf_qd2_b200.dqd2 import element_constants
    (xs, ws), (xh, wh) = gauss_legendre(24), gauss_legendre(64)
    rng = np.random.default_rng(11)
    corners = {"quad": [(-1, -1, 0), (1, -1, 0), (1, 0.9, 0), (-1, 0.9, 0)],
               "twisted": [(-1, -1, 0.1), (1, -1, -0.1), (1.1, 1, 0.1), (-1, 1, -0.1)],
               "trapezoid": [(-1, -1, 0), (1, -1, 0), (0.72, 1, 0), (-0.72, 1, 0)],
               "triangle": [(-1, -0.8, 0), (1, -0.9, 0), (0.1, 1, 0)]}[shape]
    for half in (0.02, 1.0):
        q, _ = np.linalg.qr(rng.normal(size=(3, 3)))
        rn = np.vstack([np.zeros(3), half * np.array(corners) @ q.T])
        nv = len(corners)
        ed = np.array([[0, 0, 0, 0], [1, 2, 3, 4 if nv == 4 else 0]], np.int32)
        cr, cw = element_constants(rn, ed)
        geo = np.zeros((2, 48))
        geo[1, :12], geo[1, 12:21], geo[1, 45] = cr[1].ravel(), cw[1].ravel(), nv
        c = cr[1] * (np.array([1, 1, 1, 1]) if nv == 4 else np.array([1, 1, 1, 0]))
        for tn in range(nv):
            z, e = ((-1, 1, 1, -1)[tn] / math.sqrt(3), (-1, -1, 1, 1)[tn] / math.sqrt(3)) if nv == 4 else (0, 0)
            hi = np.linalg.norm(np.stack([c[:, 1] + c[:, 3] * e, c[:, 2] + c[:, 3] * z]), 2)
            k = kr / (2.24 * hi)
            for ph in (0.0, 0.1, 1.2):
                out, ref = np.zeros(40), np.zeros(40)
                got = sh.sh_self2(geo.ctypes.data, 1, tn, k * math.cos(ph), k * math.sin(ph), xs.ctypes.data, ws.ctypes.data,
                                  xh.ctypes.data, wh.ctypes.data, out.ctypes.data, ref.ctypes.data)
                assert got == (kr < 4.0)
                if not got:
                    assert np.array_equal(out, ref)
                for lo, hi_ in ((0, 16), (16, 32), (32, 34)):
                    assert np.abs(out - ref)[lo:hi_].max() <= 2e-14 * np.abs(ref)[lo:hi_].max(), (tn, lo)
