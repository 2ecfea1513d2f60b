"""bench.py's roofline names the kernel that did the pairs, by whether the domain had a table."""


def test_roofline_follows_the_table_and_not_the_number_of_terms():
    import bench
    # a mesh with a large flat base: its pairs in one plane sum more lattice terms than all pairs have rule points
    pairs, plane = 10_000_000, 2_500_000
    terms = plane * 432 * 200
    assert terms > pairs * 432
    on = bench.regular_roofline("cone3360", dict(on=1, plane_pairs=plane, reg_smooth_ms=500.0), pairs, 0.0, terms, 3000.0, 4, 34.0)
    assert on["kernel"] == "k_reg_smooth" and on["launch_ms"] == 125.0 and on["plane_pairs_ms"] == 3000.0
    assert abs(on["achieved"] - (pairs - plane) * 432 * bench.FLOOR_OPS_PER_POINT / 0.5 / 1e12) < 1e-9
    # few terms (a small domain without a table)
    off = bench.regular_roofline("sphere384", dict(on=0, plane_pairs=0, reg_smooth_ms=0.0), 1000, 1.0, 5000, 2.0, 1, 34.0)
    assert off["kernel"] == "k_reg_periodic" and off["launch_ms"] == 2.0
    assert abs(off["achieved"] - 5000 / 2e-3 * bench.ALG_OPS_PER_TERM["sphere384"] / 1e12) < 1e-12
