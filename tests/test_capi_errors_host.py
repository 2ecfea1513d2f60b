"""Errors of the C entry points that are found before any device work."""
import ctypes as C

import numpy as np
import pytest


@pytest.mark.parametrize("lattice,want", [("degenerate", -4), ("missing", -1)])
def test_green_function_refuses_a_lattice_before_it_touches_the_device(cuda_lib_host, lattice, want):
    """bem3_qpgf with a lattice it refuses returns the lattice's error wherever it runs, a box without a
    GPU included: no copy of the caller's points is in flight when it returns."""
    import bem3_emf_qd2_b200 as B
    q = B.make_qpd(dict(k=9.0, vk=[1.0, 2.0, 8.0], vd1=[1.0, 2.0], vd2=[2.0, 4.0]))
    r, out, ret = np.ones((8, 3)), np.full((8, 4), 7.0 + 0j), np.full(8, 7, np.int32)
    rc = cuda_lib_host.bem3_qpgf(C.byref(q) if lattice == "degenerate" else None, 8, r.ctypes.data, out.ctypes.data,
                                 ret.ctypes.data, 0)
    assert rc == want
    assert (out == 7.0).all() and (ret == 7).all()
