"""bem3_last_table_stats: which kernel did a periodic domain's regular pairs, and in what time."""
import pytest

pytestmark = pytest.mark.gpu


def _stats(B, tmp_path, surf):
    from bem3_emf_qd2_b200 import meshgen
    from bem3_emf_qd2_b200.dqd2 import Problem
    cfg = dict(surfaces=[surf], media=[1.6 + 0.0j], lambda0=0.6, ni=1.33, theta=0.4, phi=2.2, d1=(1.0, 0.0), d2=(0.0, 1.0),
               e0=[(1.0, 0.0)])
    p = Problem.from_files(*meshgen.write_config("t", cfg, str(tmp_path)))
    dev = B.DeviceProblem(p)
    B.set_profiling(True)
    try:
        dev.assemble(0)
        return B.last_stats(), B.last_table_stats()
    finally:
        B.set_profiling(False)


def test_table_and_plane_pairs(cuda_lib, tmp_path):
    st, tb = _stats(cuda_lib, tmp_path, ("cone", 0.3, 0.6, -0.3, 3, 6, 12, 0.01, 7, 1, 99))
    assert tb["on"] == 1 and tb["plane_pairs"] > 0 and tb["reg_smooth_ms"] > 0.0 and st["qpgf_terms"] > 0
    assert st["reg_periodic_ms"] + tb["reg_smooth_ms"] <= st["class_ms"][1] * (1 + 1e-6)  # the rest makes the table


def test_domain_without_a_table(cuda_lib, tmp_path):
    st, tb = _stats(cuda_lib, tmp_path, ("sphere", 0.42, 1, 1, 99))  # an image 2.1 half edges away
    assert tb["on"] == 0 and tb["plane_pairs"] == 0 and st["reg_periodic_ms"] > tb["reg_smooth_ms"]
