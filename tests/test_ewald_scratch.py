"""The leaf Ewald scratch (tg_set_ewald_scratch): sums that do not fit run in
batches of leaves and ranges of vectors, with the same bits, within the bytes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _run(x, u, precision, leaf, theta, scratch):
    import tigergrav_b200 as tg
    with tg.GravitySolver(len(x), theta=theta, leaf_max=leaf, precision=precision) as s:
        s.set_ewald_scratch(scratch)
        s.set_particles(x).solve_gravity()
        report = s.memory()
        return s.get_forces(), s.tidal(u), report, s.memory()


# one leaf and one vector at a time; batches of a few leaves, ranges of vectors; several batches, all vectors
@pytest.mark.parametrize("precision,n,leaf,scratch", [("f32", 400, 16, 1), ("f64", 300, 16, 1),
                                                      ("f32", 5000, 16, 1_000_000), ("f64", 3000, 16, 1_500_000),
                                                      ("f32", 20000, 64, 1_000_000), ("f64", 9000, 40, 4_000_000)])
def test_same_bits_within_the_bytes(precision, n, leaf, scratch):
    from tigergrav_b200 import ics
    x = ics.uniform(n, n)
    u = np.random.default_rng(n + 1).standard_normal((n, 3))
    (p0, g0), j0, r0, t0 = _run(x, u, precision, leaf, 0.6, 0)
    (p1, g1), j1, r1, t1 = _run(x, u, precision, leaf, 0.6, scratch)
    assert np.array_equal(p0, p1) and np.array_equal(g0, g1) and np.array_equal(j0, j1)
    if scratch == 1:
        return
    # a buffer holds at most the bytes (at least one leaf, whose 24 chunks fit here), and a quarter more by its slack
    # (ew_part is the nodes' too)
    for full, small in ((r0, r1), (t0, t1)):
        for buf in ("ew_tpart", "ew_sf"):
            assert small[buf] <= 1.25 * scratch + 4096 < full[buf], buf


def test_argument():
    from tigergrav_b200 import _lib
    from tigergrav_b200.solver import GravitySolver
    assert _lib.lib.tg_set_ewald_scratch(None, 0) == _lib.TG_ERR_ARG
    with GravitySolver(100) as s:
        assert _lib.lib.tg_set_ewald_scratch(s.h, -1) == _lib.TG_ERR_ARG
        assert _lib.lib.tg_set_ewald_scratch(s.h, 0) == _lib.TG_OK
