"""Output matrices that start on 8-byte boundaries only, as the C ABI's `double *` promises: every
device entry point gives the same bits as into buffers that start on 16 bytes.

The domains: an interior one of 48 elements (a warp's 32 sources and a remainder), an interior one of
triangles and their open regions."""
import ctypes as C

import pytest

pytestmark = pytest.mark.gpu

KEYS = ("G", "H", "dG", "dH", "dF")


def _problems(tmp_path):
    from bem3_emf_qd2_b200 import meshgen
    from bem3_emf_qd2_b200.dqd2 import Problem
    probs = []
    for name, surf, media in (
            ("two", [("sphere", 0.3, 2, 1, 99), ("sphere", 0.2, 2, 2, 1)], [1.45 + 0.01j, 1.6]),
            ("cone", [("cone", 0.3, 0.6, -0.3, 2, 4, 8, 0.01, 7, 1, 99)], [1.6 + 0.02j])):
        cfg = dict(surfaces=surf, media=media, lambda0=0.6, ni=1.33, theta=0.4, phi=2.2, d1=(1.0, 0.0), d2=(0.0, 1.1),
                   e0=[(1.0, 0.0)])
        probs.append(Problem.from_files(*meshgen.write_config(name, cfg, str(tmp_path / name))))
    return probs


def _buffers(torch, ne, shift):
    """Outputs of a domain, each `shift` doubles into a 16-byte aligned allocation, filled with NaN."""
    n = 4 * ne
    size = dict(G=2 * n * n, H=2 * n * n, dG=4 * n * n, dH=4 * n * n, dF=3 * n)
    own = {k: torch.full((m + 2,), float("nan"), dtype=torch.float64, device="cuda") for k, m in size.items()}
    assert all(t.data_ptr() % 16 == 0 for t in own.values())
    return {k: t[shift:shift + size[k]] for k, t in own.items()}


@pytest.mark.parametrize("entry", ["bem3_assemble_domain_dev", "bem3_assemble_domain_dev_noalloc"])
def test_domain_outputs_on_8_byte_boundaries(cuda_lib, tmp_path, entry):
    import torch
    B = cuda_lib
    f = getattr(B.lib(), entry)
    f.argtypes = B.lib().bem3_assemble_domain_dev.argtypes
    for p in _problems(tmp_path):
        dp = B.DeviceProblem(p)
        for did in range(p.MN + 1):
            k, ne = complex(p.kn[did]), len(p.sid[did])
            got = []
            for shift in (0, 1):
                o = _buffers(torch, ne, shift)
                assert f(dp.geo.data_ptr(), p.Ne, dp.sids[did].data_ptr(), ne, did, int(did == 0), C.byref(dp.q), k.real,
                         k.imag, *[o[x].data_ptr() for x in KEYS], None) == 0
                torch.cuda.synchronize()
                got.append(o)
            for x in KEYS:
                assert torch.isfinite(got[0][x]).all() and torch.equal(got[0][x], got[1][x]), (did, x)


def test_batch_outputs_on_8_byte_boundaries(cuda_lib, tmp_path):
    import torch
    from bem3_emf_qd2_b200 import batch
    insts = [batch.InstanceDevice(p) for p in _problems(tmp_path)]
    got = []
    for shift in (0, 1):
        entries, outs = [], []
        for inst in insts:
            for e in inst.domain_entries():
                o = _buffers(torch, e.Ne_d, shift)
                e.G, e.H, e.dG, e.dH, e.dF = (o[x].data_ptr() for x in KEYS)
                entries.append(e)
                outs.append(o)
        batch.assemble_entries(entries)
        torch.cuda.synchronize()
        got.append(outs)
    for a, b in zip(*got):
        for x in KEYS:
            assert torch.isfinite(a[x]).all() and torch.equal(a[x], b[x]), x
