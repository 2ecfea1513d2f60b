"""The pool that the tables of a batch share: groups of domains, domains without a table among them, many small
domains, and a device without the memory for it.  Against bem3_assemble_domain_dev, as test_gpu_batch.py: 1e-13 of the
largest entry with the same plan, 1e-12 where one of them sums point by point."""
import pytest

pytestmark = pytest.mark.gpu

KEYS = ("G", "H", "dF")


def _problem(tmp_path, n, lam, period, theta=0.4, radius=0.3):
    from bem3_emf_qd2_b200 import meshgen
    from bem3_emf_qd2_b200.dqd2 import Problem
    cfg = dict(surfaces=[("sphere", radius * period, n, 1, 99)], media=[1.6 + 0.0j], lambda0=lam, ni=1.33, theta=theta,
               phi=2.2, d1=(period, 0.0), d2=(0.0, period), e0=[(1.0, 0.0)])
    return Problem.from_files(*meshgen.write_config("b", cfg, str(tmp_path / ("%d_%g_%g_%g" % (n, lam, theta, radius)))))


def _run(insts, tol):
    import torch
    from bem3_emf_qd2_b200 import batch
    b = batch.Batch(insts)
    for i in insts:
        for o in i.out:
            for k in KEYS:
                o[k].fill_(float("nan"))
    b.run()
    st = b.wait()
    assert st == [0] * len(st)
    info = b.info()
    b.close()
    got = [[{k: o[k].clone() for k in KEYS} for o in i.out] for i in insts]
    for q, i in enumerate(insts):
        i.assemble_sequential()
        torch.cuda.synchronize()
        for d, o in enumerate(i.out):
            for k in KEYS:
                err = float((got[q][d][k] - o[k]).abs().max())
                assert err <= tol * float(o[k].abs().max()), (q, d, k, err)
    return info


def test_tables_go_through_the_pool_in_groups(cuda_lib, tmp_path):
    """40 problems whose tables want 65 MB each (two groups), and between them two whose elements are too large for a
    table: those are summed point by point in the batch as alone."""
    from bem3_emf_qd2_b200 import batch
    probs = [_problem(tmp_path, 4, 0.4, 1.5, 0.1 + 0.02 * i) for i in range(40)]
    probs.insert(7, _problem(tmp_path, 1, 0.5, 1.0, radius=0.42))
    probs.insert(30, _problem(tmp_path, 1, 0.7, 1.2, radius=0.42))
    launches, nbytes = _run([batch.InstanceDevice(p, derivatives=False) for p in probs], 1e-13)
    assert launches >= 15 + 6
    assert nbytes < (2 << 30) + 42 * (2 << 20)


def test_thousands_of_small_domains_take_little_memory(cuda_lib, tmp_path):
    """4,000 open regions of 24 quads: about 0.1 MB each and the pool (25 MB each before the pool)."""
    import ctypes as C
    from bem3_emf_qd2_b200 import batch, bem3_batch_domain
    inst = batch.InstanceDevice(_problem(tmp_path, 2, 0.6, 1.0), derivatives=False)
    n = 4000
    arr = (bem3_batch_domain * n)(*([inst.domain_entries()[0]] * n))
    bound = cuda_lib.lib().bem3_batch_scratch_bytes(arr, n)
    h, nbytes = C.c_void_p(), C.c_size_t()
    assert cuda_lib.lib().bem3_batch_create(arr, n, None, C.byref(h)) == 0  # not run: the entries share their outputs
    cuda_lib.lib().bem3_batch_info(h, None, C.byref(nbytes))
    cuda_lib.lib().bem3_batch_destroy(h)
    assert nbytes.value <= bound <= (2 << 30) + n * (200 << 10)


@pytest.mark.parametrize("left", [200, 40])
def test_batch_without_memory_for_the_pool(cuda_lib, tmp_path, left):
    """Eight problems that want 520 MB of tables: with 200 MB left one table at a time, with 40 MB none."""
    import torch
    from bem3_emf_qd2_b200 import batch
    insts = [batch.InstanceDevice(_problem(tmp_path, 4, 0.4, 1.5, 0.1 + 0.1 * i), derivatives=False) for i in range(8)]
    _run(insts, 1e-13)  # loads the kernels; the matrices are now the one-domain calls'
    ref = [[{k: o[k].clone() for k in KEYS} for o in i.out] for i in insts]
    insts[0].assemble_sequential()
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    hog = torch.empty(torch.cuda.mem_get_info()[0] - (left << 20), dtype=torch.uint8, device="cuda")
    try:
        b = batch.Batch(insts)
        b.run()
        st = b.wait()
        nbytes = b.info()[1]
        b.close()
    finally:
        del hog
        torch.cuda.empty_cache()
    assert st == [0] * len(st) and nbytes < left << 20
    for i, r in zip(insts, ref):
        for o, q in zip(i.out, r):
            for k in KEYS:
                assert float((o[k] - q[k]).abs().max()) <= 1e-12 * float(q[k].abs().max()), k
