"""Host side of the pool that a batch's tables share: the library's byte bound and the wave planner."""
import ctypes as C
import math


def test_scratch_bound_counts_the_pool_once(cuda_lib_host):
    """4,000 open regions of 24 quads: about 0.2 MB each and at most 2 GB of tables; eight of them: 13 to 200 MB of table
    each.  A refused lattice counts no table."""
    from bem3_emf_qd2_b200 import bem3_batch_domain, make_qpd
    k = 2 * math.pi * 1.33 / 0.6
    q = make_qpd(dict(k=k, vk=[0.3 * k, 0.2 * k, 0.9 * k], vd1=[1.0, 0.0], vd2=[0.0, 1.0]))

    def bound(n, qd):
        arr = (bem3_batch_domain * n)()
        for e in arr:
            e.Ne, e.Ne_d, e.periodic, e.qd = 24, 24, 1, qd
        return cuda_lib_host.bem3_batch_scratch_bytes(arr, n)

    none = bound(1, type(q)())
    assert none < 200 << 10
    assert 8 * (13 << 20) <= bound(8, q) - 8 * none <= 8 * (201 << 20)
    assert bound(4000, q) <= (2 << 30) + 4000 * (200 << 10)


def test_planner_takes_the_pool_off_the_budget_once(cuda_lib_host, tmp_path):
    """With room for the pool beside the largest instance the instances count without their tables, and no wave with
    its pool exceeds the budget; without that room each counts with its own."""
    from bem3_emf_qd2_b200 import batch
    specs = [batch.InstanceSpec("sphere", 2, 1.0, 1.0 + 0.01 * i, 0.6, 0.2, 0.0, 1.5 + 0j) for i in range(12)]
    probs = batch.build_problems(specs, str(tmp_path))
    core = [batch.instance_core_bytes(p) for p in probs]
    assert all(batch.instance_bytes(p) > c + (13 << 20) for p, c in zip(probs, core))
    budget = batch.TABLE_POOL_BYTES + 4 * max(core)
    waves = [w for _, w in batch.plan(probs, budget)]
    assert sorted(i for w in waves for i in w) == list(range(12)) and len(waves) == 3
    assert all(sum(core[i] for i in w) + batch.TABLE_POOL_BYTES <= budget for w in waves)
    small = 3 * max(batch.instance_bytes(p) for p in probs)
    assert all(sum(batch.instance_bytes(probs[i]) for i in w) <= small for _, w in batch.plan(probs, small))
