"""The periodic correction's CUDA kernels at the edges of their ranges: the
FP32 path against the oracle's FP64 evaluation of the same interaction lists,
under the parity bound of helpers.arbiter_excess (1e-5 of max(|g|, g_rms / 2)
beyond the deviation of the reference's own FP32 arithmetic)."""
import numpy as np
import pytest

from helpers import arbiter_excess

pytestmark = pytest.mark.gpu


def _half_lattice(side, seed):
    """Half the points of a side^3 lattice: separations fall on 0, +-1/2 and the
    borders of the expansion table's cells."""
    rng = np.random.default_rng(seed)
    g = np.arange(side) / side
    x = np.stack(np.meshgrid(g, g, g, indexing="ij"), -1).reshape(-1, 3)
    return x[rng.permutation(len(x))[:len(x) // 2]]


CASES = {
    # name: (positions, theta, leaf_max)
    "lattice16_leaf8": (lambda: _half_lattice(16, 1), 0.7, 8),
    "lattice12_leaf1": (lambda: _half_lattice(12, 2), 0.8, 1),       # leaves of one particle, CC / CP of every length
    "uniform333_leaf5": (lambda: np.random.default_rng(3).random((333, 3)), 0.6, 5),
    "uniform5000_leaf16": (lambda: np.random.default_rng(4).random((5000, 3)), 0.45, 16),  # chunks of 128 and remainders
    "uniform70_leaf64": (lambda: np.random.default_rng(5).random((70, 3)), 0.7, 64),  # every pair is an Ewald pair
    "uniform64_leaf64": (lambda: np.random.default_rng(6).random((64, 3)), 0.7, 64),  # a single leaf
    "clump_leaf33": (lambda: (0.999 + 0.02 * np.random.default_rng(7).standard_normal((2000, 3))) % 1.0, 0.7, 33),
}


@pytest.mark.parametrize("name", list(CASES))
def test_ewald_edges(name, oracle_mod):
    import tigergrav_b200 as tg
    from tigergrav_b200 import ics
    make, theta, leaf = CASES[name]
    x = ics.double_to_pos(make())
    with tg.GravitySolver(len(x), theta=theta, leaf_max=leaf) as s:
        s.set_particles(x).solve_gravity()
        phi, g = s.get_forces()
    o = oracle_mod.Oracle(theta=theta, ewald=True, leaf_max=leaf).set_particles(x)
    o.build().multipoles().walk().evaluate()
    rphi, rg = o.forces()
    o.evaluate(fp64=True)
    phi64, g64 = o.forces()
    fx, px = arbiter_excess(g, rg, g64, phi, rphi, phi64)
    assert fx <= 0.0 and px <= 0.0, (fx, px)
