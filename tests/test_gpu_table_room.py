"""Room for the table of the smooth remainder on the GPU: a plan the room refuses, and a device without the
memory for it.  Both sum the domain point by point; tolerance 1e-12 of the largest entry, as the plain sums
differ from the table's."""
import ctypes as C
import threading

import pytest

pytestmark = pytest.mark.gpu


def _problem(tmp_path, n, lam, period):
    from bem3_emf_qd2_b200 import meshgen
    from bem3_emf_qd2_b200.dqd2 import Problem
    cfg = dict(surfaces=[("sphere", 0.3 * period, n, 1, 99)], media=[1.6 + 0.0j], lambda0=lam, ni=1.33, theta=0.4, phi=2.2,
               d1=(period, 0.0), d2=(0.0, period), e0=[(1.0, 0.0)])
    return Problem.from_files(*meshgen.write_config("s", cfg, str(tmp_path)))


def _open_region(B, p, entry="bem3_assemble_domain_dev"):
    import torch
    f = getattr(B.lib(), entry)
    f.argtypes = B.lib().bem3_assemble_domain_dev.argtypes
    dp = B.DeviceProblem(p)
    n, k = 4 * len(p.sid[0]), complex(p.kn[0])
    G = torch.full((n, n), complex("nan"), dtype=torch.complex128, device="cuda")
    H = torch.full_like(G, complex("nan"))

    def run():
        return f(dp.geo.data_ptr(), p.Ne, dp.sids[0].data_ptr(), n // 4, 0, 1, C.byref(dp.q), k.real, k.imag, G.data_ptr(),
                 H.data_ptr(), None, None, None, None)
    return run, G, H


def test_plan_that_the_static_room_refuses(cuda_lib, tmp_path):
    """96 quads at period 1.5, wavelength 0.4 want 0.8 M coefficients; the no-allocation entry has room for 0.25 M."""
    p = _problem(tmp_path, 4, 0.4, 1.5)
    run, G, H = _open_region(cuda_lib, p)
    assert run() == 0
    run2, G2, H2 = _open_region(cuda_lib, p, "bem3_assemble_domain_dev_noalloc")
    assert run2() == 0
    for a, b in ((G, G2), (H, H2)):
        assert float((a - b).abs().max()) <= 1e-12 * float(a.abs().max())


def test_assembly_without_memory_for_the_table(cuda_lib, tmp_path):
    """With 40 MB left on the device a thread's first assembly gets its lists but not the table's 65 MB."""
    import torch
    p = _problem(tmp_path, 4, 0.4, 1.5)
    run, G, H = _open_region(cuda_lib, p)
    assert run() == 0  # loads the kernels
    run2, G2, H2 = _open_region(cuda_lib, p, "bem3_assemble_domain_dev_noalloc")
    assert run2() == 0  # and those of the point-by-point sums
    torch.cuda.synchronize()
    ref = G.clone(), H.clone()
    G.fill_(complex("nan"))
    H.fill_(complex("nan"))
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    hog = torch.empty(free - (40 << 20), dtype=torch.uint8, device="cuda")
    got = []
    t = threading.Thread(target=lambda: got.append(run()))  # a thread of its own: no scratch yet
    t.start()
    t.join()
    del hog
    torch.cuda.empty_cache()
    assert got == [0]
    for a, b in zip(ref, (G, H)):
        assert float((a - b).abs().max()) <= 1e-12 * float(a.abs().max())
