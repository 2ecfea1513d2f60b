"""bem3_qpgf by a warp per point (csrc/qpgf_warp.cuh) against the host build of the serial sums: Fourier-domain
and Ewald points, both sides of the plane z = 0 and points in it, neighbouring cells, oblique lattices, point
counts around a block's four and around one pass of the host entry.

Tolerance: 1e-10 of the largest component, as the sums are held to against the reference."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LATTICES = {"square": ((1.0, 0.0), (0.0, 1.0)), "oblique": ((0.9, 0.1), (-0.35, 0.8)), "long": ((0.0, 1.7), (0.8, 0.0))}


def _qpd(lattice, k=2 * np.pi / 0.63 * 1.33):
    vk = k * np.array([np.sin(0.4) * np.cos(2.2), np.sin(0.4) * np.sin(2.2), np.cos(0.4)])
    return dict(k=k, vk=vk, vd1=np.array(LATTICES[lattice][0]), vd2=np.array(LATTICES[lattice][1]))


def _points(n, seed):
    rng = np.random.default_rng(seed)
    r = rng.uniform(-1.8, 1.8, (n, 3))
    r[::3, 2] *= 0.05
    r[::7, 2] = 0.0
    r[1::11, 2] = 3e-14
    return r


@pytest.mark.parametrize("lattice", sorted(LATTICES))
@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("n", [1, 3, 5, 517])
def test_points_equal_serial_sums(cuda_lib, devmath_host, lattice, mode, n):
    qpd = _qpd(lattice)
    r = _points(n, 10 * n + mode)
    out, ret = cuda_lib.qpgf(qpd, r, mode=mode)
    flat = np.array([qpd["k"], *qpd["vk"], *qpd["vd1"], *qpd["vd2"]])
    ref, rr = np.zeros(8 * n), np.zeros(n, np.int32)
    devmath_host.hm_qpgf(n, r.ctypes.data, flat.ctypes.data, mode, ref.ctypes.data, rr.ctypes.data)
    ref = ref.view(np.complex128).reshape(-1, 4)
    assert np.array_equal(ret > 0, rr > 0)
    ok = rr > 0
    assert ok.sum() >= 0.8 * n
    assert np.max(np.abs(out - ref)[ok] / np.abs(ref[ok]).max(axis=1, keepdims=True)) < 1e-10


def test_passes_of_many_points(cuda_lib):
    """More points than one pass of the host entry holds: the same results as the tail alone."""
    n = (1 << 18) + 3
    qpd = _qpd("square")
    r = np.tile(_points(64, 5), (n // 64 + 1, 1))[:n]
    out, ret = cuda_lib.qpgf(qpd, r, mode=0)
    o64, r64 = cuda_lib.qpgf(qpd, r[:64], mode=0)
    idx = np.arange(n) % 64
    assert np.array_equal(ret, r64[idx]) and np.array_equal(out, o64[idx], equal_nan=True)
