"""The fields' ways to the open region's Green's function (a warp per evaluation, a table for the points, plain
sums): one result whatever way a call's size takes, the memory a table takes, and calls without memory for one.

Tolerance: 1e-11 of the largest field, as the plain sums at these wave numbers differ from 64-bit sums."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _context(B, tmp_path, n, lam, period):
    from bem3_emf_qd2_b200 import meshgen
    from bem3_emf_qd2_b200.dqd2 import Problem
    cfg = dict(surfaces=[("sphere", 0.3 * period, n, 1, 99)], media=[1.6 + 0.0j], lambda0=lam, ni=1.33, theta=0.4, phi=2.2,
               d1=(period, 0.0), d2=(0.0, period), e0=[(1.0, 0.0)])
    p = Problem.from_files(*meshgen.write_config("f", cfg, str(tmp_path)))
    ctx = B.Context(p)
    rng = np.random.default_rng(1)
    bv = []
    for d in range(2):
        shape = (len(p.sid[d]) + 1, 4)
        bv.append({k: rng.normal(size=shape + (m,)) + 1j * rng.normal(size=shape + (m,))
                   for k, m in (("U", 4), ("dU", 4), ("E", 3), ("dE", 3), ("H", 3), ("dH", 3))})
    ctx.set_boundary_values(bv)
    return ctx


def _points(rng, n, period, top):
    r = rng.uniform(-0.9 * period, 0.9 * period, (n, 3))
    r[:, 2] = np.where(r[:, 2] < 0, -1, 1) * rng.uniform(0.4 * period, top, n)
    return r


@pytest.mark.parametrize("lam,period,type_", [(0.6328, 1.0, 0), (0.6328, 1.0, 1), (0.4, 1.5, 1), (0.8, 0.8, 2)])
def test_one_result_for_every_number_of_points(cuda_lib, tmp_path, lam, period, type_):
    """1,500 points at once (a table, several CTAs of elements) and the first 1, 7 and 60 of them alone."""
    ctx = _context(cuda_lib, tmp_path, 5, lam, period)
    r = _points(np.random.default_rng(2), 1500 if type_ < 2 else 40, period, 1.2 * period)
    E, H, _ = ctx.field(r, type_, True)
    for n in (1, 7, 60):
        if n > len(r):
            continue
        e, h, _ = ctx.field(r[:n], type_, True)
        assert np.abs(e - E[:n]).max() <= 1e-11 * np.abs(E).max() and np.abs(h - H[:n]).max() <= 1e-11 * np.abs(H).max()


@pytest.mark.parametrize("type_", [0, 1])
def test_points_in_the_plane_of_the_rules_points(cuda_lib, tmp_path, type_):
    """A probe plane through the middle of a sphere with an odd number of element rows, where rule points share the
    field points' height: few of them by warps, many by a table, against the plane 1e-9 periods above."""
    ctx = _context(cuda_lib, tmp_path, 5, 0.6328, 1.0)
    rng = np.random.default_rng(4)
    a = rng.uniform(0, 2 * np.pi, 1500)
    r = np.stack([0.45 * np.cos(a), 0.45 * np.sin(a), np.zeros(1500)], 1)
    up = r + np.array([0.0, 0.0, 1e-9])
    E, H, _ = ctx.field(up, type_, True)
    for n in (3, 1500):
        e, h, _ = ctx.field(r[:n], type_, True)
        # the fields change by k 1e-9 or so; in the plane the reference's sums stop on rounding noise (6e-5 of G)
        assert np.abs(e - E[:n]).max() <= 1e-4 * np.abs(E).max() and np.abs(h - H[:n]).max() <= 1e-4 * np.abs(H).max()


def test_partial_sums_in_several_chunks(cuda_lib, tmp_path):
    """More points than one launch takes (256 MB of partial sums, 312 bytes a point at 384 elements): 900,000 points
    against the same in halves."""
    ctx = _context(cuda_lib, tmp_path, 8, 0.6328, 1.0)
    r = _points(np.random.default_rng(3), 900000, 1.0, 0.6)
    E, H, did = ctx.field(r, 0, False)
    half = [ctx.field(r[s], 0, False) for s in (slice(0, 450001), slice(450001, None))]
    assert np.array_equal(np.concatenate([half[0][2], half[1][2]]), did)
    for k, full in ((0, E), (1, H)):
        assert np.abs(np.concatenate([half[0][k], half[1][k]]) - full).max() <= 1e-11 * np.abs(full).max()


def _in_a_thread(f):
    got = []

    def run():
        try:
            got.append(f())
        except BaseException as e:
            got.append(e)
    t = threading.Thread(target=run)
    t.start()
    t.join()
    if isinstance(got[0], BaseException):
        raise got[0]
    return got[0]


def test_table_takes_the_memory_it_needs(cuda_lib, tmp_path):
    """A thread's first call with one point of rule 2 on 54 quads: its table is small (it was 100 MB for every
    call)."""
    import torch
    ctx = _context(cuda_lib, tmp_path, 3, 0.6328, 1.0)
    r = np.array([[0.1, 0.2, 0.45]])
    ctx.field(r, 2, True)  # loads the kernels

    def first():
        torch.cuda.synchronize()
        before = torch.cuda.mem_get_info()[0]
        ctx.field(r, 2, True)
        return before - torch.cuda.mem_get_info()[0]
    assert _in_a_thread(first) < 40 << 20


def test_fields_without_memory_for_the_table(cuda_lib, tmp_path):
    """With 24 MB left on the device a thread's first call takes no table and gives the same fields."""
    import torch
    ctx = _context(cuda_lib, tmp_path, 4, 0.4, 1.5)
    r = _points(np.random.default_rng(5), 2000, 1.5, 4.0)
    E, H, _ = ctx.field(r, 1, True)
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    hog = torch.empty(free - (24 << 20), dtype=torch.uint8, device="cuda")
    try:
        e, h, _ = _in_a_thread(lambda: ctx.field(r, 1, True))
    finally:
        del hog
        torch.cuda.empty_cache()
    assert np.abs(e - E).max() <= 1e-11 * np.abs(E).max() and np.abs(h - H).max() <= 1e-11 * np.abs(H).max()
