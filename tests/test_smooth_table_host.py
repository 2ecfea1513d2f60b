"""The samples and the table of the smooth remainder as the assembly makes them (csrc/smooth.cuh,
csrc/assemble_smooth.cuh), on the host build."""
import ctypes as C
import math
import os
import subprocess

import numpy as np
import pytest

from conftest import BUILD, REPO


@pytest.fixture(scope="module")
def st():
    os.makedirs(BUILD, exist_ok=True)
    so = os.path.join(BUILD, "libsmooth_table_host.so")
    native, hdr = os.path.join(REPO, "tests", "native"), os.path.join(REPO, "bem3_emf_qd2_b200", "csrc")
    subprocess.run(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-I" + hdr,
                    os.path.join(native, "smooth_table_host.cpp"), "-o", so], check=True)
    lib = C.CDLL(so)
    vp, i, d = C.c_void_p, C.c_int, C.c_double
    lib.st_real.argtypes = [vp, vp, d, d, vp, vp]
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
