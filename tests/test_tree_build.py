"""The tree build at the width where a level leaves the one-cluster kernel (131072
nodes) for passes over the whole GPU, and back; and where the node arrays turn
out too small in one or the other: nodes identical to the oracle's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _uniform(n, seed):
    return np.random.default_rng(seed).random((n, 3))


def _lattice(a, b, c):
    g = np.stack(np.meshgrid((np.arange(a) + 0.5) / a, (np.arange(b) + 0.5) / b, (np.arange(c) + 0.5) / c,
                             indexing="ij"), -1)
    return g.reshape(-1, 3)


def _pairs(n, sep, seed):
    """n points, each with a partner at `sep`: long chains of nodes with one empty child"""
    x = _uniform(n, seed)
    return np.concatenate([x, (x + sep / np.sqrt(3.0)) % 1.0])


def _clump(n, k, seed):
    x = _uniform(n, seed)
    x[:k] = 0.7 + 0.02 * np.random.default_rng(seed + 1).random((k, 3))
    return x


CASES = {
    # name: (positions, leaf_max)
    "widest_narrow": (lambda: _lattice(64, 64, 32), 1),           # the last level has 131072 nodes, all leaves
    "wide": (lambda: _uniform(300000, 2), 1),                     # several wide levels, then narrow ones
    "wide_last": (lambda: _lattice(64, 64, 64), 1),               # and 262144
    "wide_then_deep": (lambda: _clump(280000, 9000, 4), 1),       # levels below the wide ones in the cluster again
    "wide_regrow": (lambda: _pairs(80000, 2.0 ** -11, 5), 1),     # more nodes than 4 n / leaf_max, in wide levels
    "narrow_regrow": (lambda: _pairs(3000, 2.0 ** -16, 6), 1),    # and in narrow ones
}


@pytest.mark.parametrize("name", list(CASES))
def test_wide_levels(name, oracle_mod):
    import tigergrav_b200 as tg
    from tigergrav_b200 import ics
    make, leaf = CASES[name]
    x = ics.double_to_pos(make())
    o = oracle_mod.Oracle(theta=0.7, ewald=True, leaf_max=leaf).set_particles(x)
    on = o.build().multipoles().nodes()
    with tg.GravitySolver(len(x), theta=0.7, leaf_max=leaf) as s:
        s.set_particles(x)
        for _ in range(2):  # the second build has the first one's arrays
            gn = s.build().multipoles().nodes()
            for k in ("boxid", "level", "child0", "parent", "pbegin", "pend"):
                np.testing.assert_array_equal(gn[k], on[k], err_msg=k)
