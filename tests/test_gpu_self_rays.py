"""Interior self pairs on the GPU by both ray rules, 24 points in ln r and, past |k K| r = 4, 64 points in r, against
the host build's 64 points.

Tolerance: 1e-11 of the row's largest self entry of each kind, as the host build differs from the reference."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", ["sphere", "cone"])
@pytest.mark.parametrize("n,lam,index,past", [(4, 0.8, 1.5 + 0.02j, False), (1, 0.25, 3.2 + 0.05j, True)])
def test_self_pairs_by_both_ray_rules(cuda_lib, devmath_host, tmp_path, shape, n, lam, index, past):
    from bem3_emf_qd2_b200 import meshgen
    from bem3_emf_qd2_b200.dqd2 import Problem
    B = cuda_lib
    surf = ("sphere", 0.3, n, 1, 99) if shape == "sphere" else ("cone", 0.3, 0.6, -0.3, n, 2 * n, 4 * n, 0.01, 7, 1, 99)
    cfg = dict(surfaces=[surf], media=[index], lambda0=lam, ni=1.0, theta=0.4, phi=2.2, d1=(1.0, 0.0), d2=(0.0, 1.0),
               e0=[(1.0, 0.0)])
    p = Problem.from_files(*meshgen.write_config("s", cfg, str(tmp_path)))
    k = complex(p.kn[1])
    reach = [2.24 * abs(k) * np.linalg.norm(p.cr[s][:, 1:3], 2) for s in range(1, p.Ne + 1)]
    assert min(reach) > 8.0 if past else max(reach) < 4.0
    M = B.assemble_domain(p, 1)
    geo = B.MeshArrays(p).packed()
    (xl, wl), (xh, wh) = B.gauss_legendre(12), B.gauss_legendre(64)
    for t, sd in list(enumerate(p.sid[1]))[::max(1, len(p.sid[1]) // 12)]:
        for tn in range(int(p.nv[abs(sd)])):
            out = np.zeros(54)
            devmath_host.hm_self_interior(geo.ctypes.data, int(sd), tn, k.real, k.imag, xl.ctypes.data, wl.ctypes.data,
                                          xh.ctypes.data, wh.ctypes.data, out.ctypes.data)
            c = out[0::2] + 1j * out[1::2]
            row, cols = 4 * t + tn, slice(4 * t, 4 * t + 4)
            h = M["H"][row, cols].copy()
            h[tn] -= M["dF"][row, 0]  # the row sum of F sits on the diagonal
            for got, ref in ((M["G"][row, cols], c[0:4]), (h, c[4:8]), (M["dG"][2 * row, cols], c[9:13]),
                             (M["dH"][2 * row, cols], c[13:17])):
                assert np.abs(got - ref).max() <= 1e-11 * max(np.abs(ref).max(), np.abs(c[0:4]).max()), (t, tn)
