"""The open region's matrices with the tabulated remainder on the GPU (csrc/assemble_smooth.cuh) against
the host build of the plain lattice sums, at sampled pairs: lattices of every orientation, quads and
triangles, shifted and near-singular pairs, pairs in one plane, element counts around the four sources of
a warp, and a domain whose elements are too large for a table.

Tolerance: 1e-12 of the row block's largest entry, as the plain sums differ from the reference."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _problem(shape, n, lattice, lam, tmp_path):
    from bem3_emf_qd2_b200 import meshgen
    from bem3_emf_qd2_b200.dqd2 import Problem
    d1, d2 = lattice
    r = 0.3 * min(math.hypot(*d1), math.hypot(*d2))
    surf = ("sphere", r, n, 1, 99) if shape == "sphere" else ("cone", r, 2 * r, -r, n, 2 * n, 4 * n, 0.01, 7, 1, 99)
    cfg = dict(surfaces=[surf], media=[1.6 + 0.02j], lambda0=lam, ni=1.33, theta=0.4, phi=2.2, d1=d1, d2=d2, e0=[(1.0, 0.0)])
    return Problem.from_files(*meshgen.write_config("m", cfg, str(tmp_path)))


@pytest.mark.parametrize("shape,n,lattice,lam,drop", [
    ("sphere", 4, ((1.0, 0.0), (0.0, 1.0)), 0.6, 0), ("sphere", 4, ((0.0, 1.1), (1.0, 0.0)), 0.5, 1),
    ("sphere", 3, ((1.0, 0.1), (0.3, 0.9)), 0.7, 2), ("cone", 3, ((0.9, 0.0), (0.45, 0.7794)), 0.7, 3),
    ("cone", 3, ((0.8, 0.0), (0.0, 1.5)), 0.45, 0), ("sphere", 1, ((1.0, 0.0), (0.0, 1.0)), 0.4, 0)])
def test_matrices_equal_plain_lattice_sums(cuda_lib, devmath_host, tmp_path, shape, n, lattice, lam, drop):
    import torch
    B = cuda_lib
    p = _problem(shape, n, lattice, lam, tmp_path)
    if drop:  # fewer elements: counts that are no multiple of four
        p.sid = [s[:-drop] for s in p.sid]
    ne = len(p.sid[0])
    dev = B.DeviceProblem(p)
    for t in (dev.G, dev.H, dev.dF):
        t.fill_(float("nan"))
    dev.assemble(0)
    N = 4 * ne
    G = dev.G.reshape(-1)[:N * N].view(N, N).cpu().numpy()
    H = dev.H.reshape(-1)[:N * N].view(N, N).cpu().numpy()
    assert np.isfinite(G).all() and np.isfinite(H).all() and np.isfinite(dev.dF.cpu().numpy()[:N]).all()
    G2, H2 = dev.G.clone(), dev.H.clone()
    dev.assemble(0)
    assert torch.equal(dev.G, G2) and torch.equal(dev.H, H2)
    geo = B.MeshArrays(p).packed()
    q = p.qpd
    qpd = np.array([q["k"], *q["vk"], *q["vd1"], *q["vd2"]])
    tabs = {m: B.gauss_legendre(m) for m in (12, 64)}
    rng = np.random.default_rng(3)
    rows = rng.choice(ne, 6, replace=False)
    seen = 0
    for t in rows:
        nv = int(p.nv[p.sid[0][t]])
        block = slice(4 * t, 4 * t + nv)
        sc_g, sc_h = np.abs(G[block]).max(), np.abs(H[block]).max()
        near = np.argsort(np.linalg.norm(p.cr[p.sid[0]][:, :, 0] - p.cr[p.sid[0][t], :, 0], axis=1))[1:4]
        for s in sorted(set(near) | set(rng.choice(ne, 6, replace=False)) | {0, ne - 1}):
            if s == t:
                continue
            for tn in range(nv):
                out = np.zeros(54)
                args = [geo.ctypes.data, int(p.sid[0][t]), tn, int(p.sid[0][s]), 1, 1.0, 0.0, qpd.ctypes.data]
                for m in (12, 64):
                    x, w = (np.ascontiguousarray(v) for v in tabs[m])
                    if not devmath_host.hm_pair_regular(*args, m, x.ctypes.data, w.ctypes.data, out.ctypes.data):
                        break
                c = out[0::2] + 1j * out[1::2]
                if shape == "cone" and abs(p.cr[p.sid[0][s], 2, 0] - p.ren[p.sid[0][t], tn, 2]) < 1e-9:
                    tol = 1e-4  # one plane: the stop rule of these sums decides on rounding noise
                else:
                    tol = 1e-12
                assert np.abs(G[4 * t + tn, 4 * s:4 * s + 4] - c[0:4]).max() <= tol * sc_g, (t, tn, s)
                assert np.abs(H[4 * t + tn, 4 * s:4 * s + 4] - c[4:8]).max() <= tol * sc_h, (t, tn, s)
                seen += 1
    assert seen > 50
