"""The samples and the table of the smooth remainder as the assembly makes them (csrc/smooth.cuh,
csrc/assemble_smooth.cuh), on the host build."""
import ctypes as C
import math
import os
import subprocess

import numpy as np
import pytest

import test_smooth_host as pairs
from conftest import REPO


@pytest.fixture(scope="module")
def st(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("table") / "libsmooth_table_host.so")
    native, hdr = os.path.join(REPO, "tests", "native"), os.path.join(REPO, "bem3_emf_qd2_b200", "csrc")
    subprocess.run(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-I" + hdr,
                    os.path.join(native, "smooth_table_host.cpp"), "-o", so], check=True)
    lib = C.CDLL(so)
    vp, i, d = C.c_void_p, C.c_int, C.c_double
    lib.st_real.argtypes = [vp, vp, d, d, vp, vp]
    lib.st_sums.argtypes = [vp, vp, i, vp]
    lib.st_capacity.argtypes = [vp, i]
    lib.st_plan_size.argtypes = [vp, vp, i, d]
    lib.st_capacity.restype = lib.st_plan_size.restype = d
    lib.st_reach.argtypes = [vp, i, i, vp, vp]
    lib.st_reach.restype = d
    lib.st_nq.argtypes = [d, d, d, d, i]
    lib.st_pair.argtypes = [vp, i, i, i, i, vp, vp, vp]
    lib.sh_plan.argtypes = [vp, vp, i, d, i, vp]
    return lib


@pytest.mark.parametrize("lam", [0.4, 0.8, 5.0])
def test_samples_close_to_an_image_keep_their_digits(st, lam):
    """Real-space part of a sample at 1e-12 to 0.3 from the origin's image and from another one of its block,
    against 40-digit sums.  There the term and the image taken off are both 1 / (4 pi R).  Tolerance: 32
    roundings of the size that is left, the other terms' sum and 1 / (4 pi ve) e^{(k ve)^2} of the image."""
    import mpmath as mp
    mp.mp.dps = 40
    k = 2 * math.pi * 1.33 / lam
    lat = np.array([k, 0.35 * k, -0.2 * k, 1.0, 0.0, 0.3, 0.9])
    rng = np.random.default_rng(int(10 * lam))
    for at in ((0.0, 0.0), (1.0, 0.0)):
        for dist in (0.0, 1e-12, 1e-7, 1e-3, 0.02, 0.05, 0.1, 0.3):
            u = rng.normal(size=3)
            r = np.array([*at, 0.0]) + dist * u / np.linalg.norm(u)
            out, ve = np.zeros(2), C.c_double()
            assert st.st_real(lat.ctypes.data, r.ctypes.data, -1.0, -1.0, out.ctypes.data, C.byref(ve)) == 1
            kk, v = mp.mpf(float(lat[0])), mp.mpf(ve.value)
            ref, size = mp.mpc(0), mp.mpf(0)
            for a in range(-4, 5):
                for b in range(-4, 5):
                    x = mp.mpf(float(r[0])) + a + b * mp.mpf(float(lat[5]))
                    y = mp.mpf(float(r[1])) + b * mp.mpf(float(lat[6]))
                    R = mp.sqrt(x * x + y * y + mp.mpf(float(r[2])) ** 2)
                    if R < mp.mpf(10) ** -15:
                        R = mp.mpf(10) ** -15  # the limit
                    z = mp.mpc(kk * v, R / (2 * v))
                    t = mp.re(mp.exp(mp.mpc(0, -1) * kk * R) * mp.erfc(-1j * z))
                    image = a in (0, -1) and b in (0, -1)
                    if image:
                        t = t - mp.expj(kk * R)
                    ph = mp.expj(mp.mpf(float(lat[1])) * (a + b * mp.mpf(float(lat[5]))) + mp.mpf(float(lat[2])) * b * mp.mpf(float(lat[6])))
                    ref += ph * t / (4 * mp.pi * R)
                    size += min(1 / R, 1 / v) / (4 * mp.pi) * mp.exp((kk * v) ** 2) if image else abs(t) / (4 * mp.pi * R)
            assert abs(complex(*out) - complex(ref)) <= 32 * 1.1e-16 * float(size), (at, dist)


def _sphere(n, lam, lattice):
    """Geometry records of a cube-sphere of 6 n^2 quads and the lattice's seven numbers."""
    from bem3_emf_qd2_b200 import meshgen
    from bem3_emf_qd2_b200.dqd2 import element_constants
    nodes = meshgen._Nodes()
    els = meshgen.cube_sphere(nodes, 0.3 * min(lattice[0], lattice[3]), n)
    rn = np.vstack([np.zeros(3), np.array(nodes.pts)])
    ed = np.vstack([np.zeros(4, int), np.array(els)]).astype(np.int32)
    cr, cw = element_constants(rn, ed)
    geo = np.zeros((len(ed), 48))
    geo[1:, 0:12], geo[1:, 12:21], geo[1:, 45] = cr[1:].reshape(-1, 12), cw[1:].reshape(-1, 9), 4
    g = 1 / math.sqrt(3)
    for j, (z, e) in enumerate(((-g, -g), (g, -g), (g, g), (-g, g))):
        geo[:, 21 + 3 * j:24 + 3 * j] = cr[:, :, 0] + cr[:, :, 1] * z + cr[:, :, 2] * e + cr[:, :, 3] * z * e
    k = 2 * math.pi * 1.33 / lam
    return np.ascontiguousarray(geo), np.array([k, 0.35 * k, -0.2 * k, *lattice])


@pytest.mark.parametrize("n,lam,lattice", [
    (4, 0.6, (1.0, 0.0, 0.0, 1.0)), (4, 3.0, (0.8, 0.0, 0.0, 1.5)), (8, 3.0, (1.0, 0.0, 0.0, 1.0)),
    (4, 10.0, (1.0, 0.0, 0.0, 1.0)), (4, 50.0, (1.0, 0.0, 0.0, 1.0)), (4, 2000.0, (1.0, 0.0, 0.4, 0.9))])
def test_gradients_of_the_table_where_the_wavelength_is_above_the_period(st, n, lam, lattice):
    """H of sampled pairs against 64-bit sums.  Tolerance: 8 roundings (1.8e-15) of the size of the parts the
    sum consists of, the normal weight W times the gradients of the four nearest images, 1 / (4 pi R^2), and of
    the wave of order (0, 0), 1 / (2 |cell|); above k = 2 pi / period the images' gradients are (1 + k R) as large."""
    from bem3_emf_qd2_b200 import gauss_legendre
    geo, lat = _sphere(n, lam, lattice)
    ne, info = len(geo) - 1, np.zeros(8, np.int32)
    assert st.sh_plan(lat.ctypes.data, geo.ctypes.data, ne, 4.0 * ne * ne, 0, info.ctypes.data) == 1 and info[0] == 1
    x, w = gauss_legendre(12)
    d1, d2 = np.array([*lattice[:2], 0]), np.array([*lattice[2:], 0])
    rng = np.random.default_rng(n)
    for _ in range(40):
        t, s = rng.choice(ne, 2, replace=False) + 1
        tn = int(rng.integers(4))
        out = np.zeros(19)
        st.st_pair(geo.ctypes.data, t, tn, s, 12, x.ctypes.data, w.ctypes.data, out.ctypes.data)
        _, ref = pairs._reference(lat, geo, t, tn, s)
        v = geo[s, [0, 4, 8]] - geo[t, 21 + 3 * tn:24 + 3 * tn]
        R = np.sort([np.linalg.norm(v + a * d1 + b * d2) for a in (-1, 0, 1) for b in (-1, 0, 1)])[:4]
        size = ((1 + lat[0] * R) / (4 * math.pi * R * R)).sum() + 0.5 / abs(lattice[0] * lattice[3] - lattice[1] * lattice[2])
        size *= np.linalg.norm(geo[s, 12:21:3])
        H = out[8:16:2] + 1j * out[9:16:2]
        assert np.abs(H - ref).max() <= 1.8e-15 * size, (t, tn, s)


def _gauss(n):
    """Nodes and weights of the n-point rule in extended precision."""
    x = np.cos(np.pi * (np.arange(n) + 0.75) / (n + 0.5)).astype(np.longdouble)
    for _ in range(8):
        p, q = np.ones(n, np.longdouble), np.zeros(n, np.longdouble)
        for j in range(1, n + 1):
            p, q = ((2 * j - 1) * x * p - (j - 1) * q) / np.longdouble(j), p
        d = n * (x * p - q) / (x * x - 1)
        x = x - p / d
    return x, 2 / ((1 - x * x) * d * d)


@pytest.mark.parametrize("shape", ["square", "rhombus", "rectangle", "triangle", "right", "obtuse"])
@pytest.mark.parametrize("n", range(4, 17))
def test_smooth_rule_at_the_nearest_image_it_accepts(st, shape, n):
    """The rule that smooth_nq gives with an image as near as it accepts for n points, against 56 points in
    extended precision: 1 / R and r / R^3 times the shape functions, the image in any direction.  Tolerance:
    SMT_QTOL = 5e-16 of the integrands' sizes, the bound smooth_nq states.  Nearer images take more points, and
    below the last bound there is no rule."""
    near, far = 1.5, 1000.0
    tri = int(shape in ("triangle", "right", "obtuse"))
    assert st.st_nq(1e-3, 1.0, near, 0.0, tri) == 0
    for _ in range(60):
        mid = math.sqrt(near * far)
        got = st.st_nq(1e-3, 1.0, mid, 0.0, tri)
        near, far = (near, mid) if 0 < got <= n else (mid, far)
    s3 = np.sqrt(np.longdouble(3))

    def rule(m):
        x, w = _gauss(m)
        if not tri:
            a, b = np.meshgrid(x, x, indexing="ij")
            W = np.outer(w, w)
            N = np.stack([(1 - s3 * a) * (1 - s3 * b), (1 + s3 * a) * (1 - s3 * b), (1 + s3 * a) * (1 + s3 * b), (1 - s3 * a) * (1 + s3 * b)]) / 4
            ang = {"square": 90, "rhombus": 60, "rectangle": 90}[shape]
            h = 0.4 if shape == "rectangle" else 1.0
            P = np.stack([a + math.cos(math.radians(ang)) * h * b, math.sin(math.radians(ang)) * h * b, 0 * a])
        else:  # collapsed square, side 2
            x1, w1 = _gauss(m + 1)
            a, b = np.meshgrid(x1, x, indexing="ij")
            u, v = (1 + a) / 2, (1 + b) / 2
            W = np.outer(w1, w) * u
            z, e = -0.5 + 1.5 * u - 1.5 * u * v, s3 * (-0.5 + 0.5 * u + 0.5 * u * v)
            N = np.stack([1 - 2.5 * (z + s3 * e), 1 + 5 * z, 1 - 2.5 * (z - s3 * e)]) / 3
            V = {"triangle": [(-1, -1), (1, -1), (0, 3 ** 0.5 - 1)], "right": [(-1, 0), (1, 0), (0, 1)],
                 "obtuse": [(-1, 0), (1, 0), (0, 0.4)]}[shape]  # longest edge 2
            V = np.array(V) - np.mean(V, 0)
            w0, w1_, w2 = (1 - z - s3 * e) / 3, (1 + 2 * z) / 3, (1 - z + s3 * e) / 3
            P = np.stack([w0 * V[0, q] + w1_ * V[1, q] + w2 * V[2, q] for q in (0, 1)] + [0 * z])
        v = P[None] - at[:, :, None, None]
        R = np.sqrt((v * v).sum(1))
        f = np.concatenate([(1 / R)[:, None], v / R[:, None] ** 3], 1)
        return np.einsum("mfij,kij,ij->mfk", f, N, W), (W / R).sum((1, 2)), (W / R ** 2).sum((1, 2))

    ph, th = np.linspace(0, 2 * np.pi, 37), np.linspace(0, np.pi / 2, 5)
    at = np.array([[np.sin(t) * np.cos(p), np.sin(t) * np.sin(p), np.cos(t)] for t in th for p in ph]).astype(np.longdouble) * far
    got, ref = rule(n)[0], rule(56)
    err = np.abs(got - ref[0]).max(2)
    assert (err[:, 0] <= 5e-16 * ref[1]).all() and (err[:, 1:].max(1) <= 5e-16 * ref[2]).all()


@pytest.mark.parametrize("tri", [False, True])
def test_reach_bounds_every_row(st, tri):
    """The interior kernel's bound of its rows' half lengths, which its Taylor sums' range is tested against,
    on elements whose one direction is much longer than the other."""
    rng = np.random.default_rng(17)
    a = np.linspace(-1.0, 1.0, 41)
    for trial in range(60):
        geo = np.zeros((2, 48))
        cr = rng.normal(size=(3, 4)) * np.array([1.0, *10.0 ** rng.uniform(-3, 0, 3)])
        if tri:
            cr[:, 3] = 0.0
        geo[1, :12], geo[1, 45] = cr.ravel(), 3 if tri else 4
        longest = C.c_double()
        reach = st.st_reach(geo.ctypes.data, 1, 41, a.ctypes.data, C.byref(longest))
        assert longest.value <= reach * (1 + 1e-12), trial


def _cone(n, r):
    """Geometry records of a triangulated cone, height 2 r."""
    from bem3_emf_qd2_b200 import meshgen
    from bem3_emf_qd2_b200.dqd2 import element_constants
    nodes = meshgen._Nodes()
    els = meshgen.cone(nodes, r, 2 * r, -r, n, 2 * n, 4 * n, 0.01, 3)
    rn = np.vstack([np.zeros(3), np.array(nodes.pts)])
    ed = np.array([[0, 0, 0, 0]] + [list(e) + [0] * (4 - len(e)) for e in els], np.int32)
    cr, cw = element_constants(rn, ed)
    geo = np.zeros((len(ed), 48))
    geo[1:, 0:12], geo[1:, 12:21], geo[1:, 45] = cr[1:].reshape(-1, 12), cw[1:].reshape(-1, 9), 3
    return np.ascontiguousarray(geo)


@pytest.mark.parametrize("shape,n", [("sphere", 2), ("sphere", 3), ("sphere", 4), ("sphere", 5), ("sphere", 6), ("sphere", 7),
                                     ("sphere", 10), ("cone", 2), ("cone", 3), ("cone", 4)])
@pytest.mark.parametrize("hexagonal", [False, True])
@pytest.mark.parametrize("lam,period", [(0.8, 0.8), (0.6328, 1.0), (0.5, 1.2), (0.4, 1.5)])
def test_table_has_room_whatever_the_number_of_elements(st, shape, n, lam, period, hexagonal):
    """Meshes of every size keep their table over the whole range of wavelengths and periods: the room the host
    gives it holds a plan wherever the elements admit one at all."""
    lattice = (period, 0.0, 0.5 * period, 0.866 * period) if hexagonal else (period, 0.0, 0.0, period)
    geo, lat = _sphere(n, lam, lattice)
    if shape == "cone":
        geo = _cone(n, 0.3 * min(lattice[0], lattice[3]))
        lat[0] /= 1.33
    ne = len(geo) - 1
    cap = st.st_capacity(lat.ctypes.data, ne)
    assert 0 < cap <= 1 << 22
    assert 0 < st.st_plan_size(lat.ctypes.data, geo.ctypes.data, ne, cap) <= cap


def test_plan_is_refused_by_the_capacity_or_fits_it(st):
    """A smaller room gives a plan of a higher degree with fewer coefficients, a still smaller one none."""
    geo, lat = _sphere(8, 0.6328, (1.0, 0.0, 0.0, 1.0))
    free = st.st_plan_size(lat.ctypes.data, geo.ctypes.data, 384, 1e12)
    assert st.st_plan_size(lat.ctypes.data, geo.ctypes.data, 384, free + 4) == free
    less = st.st_plan_size(lat.ctypes.data, geo.ctypes.data, 384, free - 1)
    assert 0 < less < free
    assert st.st_plan_size(lat.ctypes.data, geo.ctypes.data, 384, 1 << 15) == 0


@pytest.mark.parametrize("seed", range(6))
def test_sums_with_the_propagating_orders_first_reach_far_points(st, seed):
    """The lattice sums that take the propagating orders first, at heights of 0.001 to 8 over seeded lattices (sides
    1 : 0.2 to 1 : 5, skewed, wavelengths 0.35 to 4), against 64-bit sums.  At far points the evanescent orders close to
    grazing lie behind rows of propagating ones, which must not end the walk.  Tolerance: 1e-11 of the largest
    value, as the plain sums' terms reach e^3 times a sum that may be small."""
    rng = np.random.default_rng(seed)
    for _ in range(25):
        d1, asp, sk = rng.uniform(0.5, 2), math.exp(rng.uniform(-1.6, 1.6)), rng.uniform(-0.5, 0.5)
        k = 2 * math.pi * rng.choice([1, 1.33]) / math.exp(rng.uniform(math.log(0.35), math.log(4)))
        th, ph = rng.uniform(0.001, 1.2), rng.uniform(0, 2 * math.pi)
        if k * k * d1 * d1 * asp > 600:
            continue
        lat = np.array([k, k * math.sin(th) * math.cos(ph), k * math.sin(th) * math.sin(ph), d1, 0, sk * d1, asp * d1])
        r = np.concatenate([rng.uniform(-1.5, 1.5, (5, 2)), np.exp(rng.uniform(math.log(1e-3), math.log(8), (5, 1)))], 1)
        r[::2, 2] *= -1
        r, out = np.ascontiguousarray(r), np.zeros((5, 8))
        assert st.st_sums(lat.ctypes.data, r.ctypes.data, 5, out.ctypes.data) >= 0
        ref = pairs._green(lat, r)
        assert (np.abs(out.view(complex) - ref).max(1) <= 1e-11 * np.abs(ref).max(1)).all(), (lat, r)
