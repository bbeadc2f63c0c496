"""The walk's leaf drain where the leaves of a level are rare, common or end in
the middle of a warp's claim: the eight lists identical to the oracle's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _spread(clump, alone, seed):
    """`clump` points within 1e-3 and `alone` in the rest of the box: leaves on many levels."""
    rng = np.random.default_rng(seed)
    c = 0.3 + 1e-3 * rng.random((clump, 3))
    return np.concatenate([c, rng.random((alone, 3))])


CASES = {
    # name: (positions, theta, leaf_max, ewald)
    "one_alone": (lambda: _spread(4000, 1, 1), 0.7, 16, True),
    "few_alone": (lambda: _spread(3000, 77, 2), 0.5, 8, True),
    "many_alone": (lambda: _spread(500, 2500, 3), 0.7, 1, False),
    "single_leaf": (lambda: _spread(30, 3, 4), 0.7, 64, True),
}


@pytest.mark.parametrize("name", list(CASES))
def test_drain_lists(name, oracle_mod):
    import tigergrav_b200 as tg
    from tigergrav_b200 import ics
    make, theta, leaf, ewald = CASES[name]
    x = ics.double_to_pos(make())
    o = oracle_mod.Oracle(theta=theta, ewald=ewald, leaf_max=leaf).set_particles(x)
    o.build().multipoles().walk()
    with tg.GravitySolver(len(x), theta=theta, ewald=ewald, leaf_max=leaf) as s:
        s.set_particles(x).solve_gravity()
        for k in ("CC_D", "CP_D", "CC_E", "CP_E", "PC_D", "PP_D", "PC_E", "PP_E"):
            for got, want in zip(s.list(k), o.list(k)):
                np.testing.assert_array_equal(got, want, err_msg=k)
