"""Potentials near zero of small periodic boxes, where every pair is a PP Ewald
pair or nearly so: the mean over the particles of the FP32 path's phi stays
within 4e-7 of the oracle's in the reference's arithmetic.  Both lie below the FP64
sums: the oracle by the mean error of its erfc, 5.3e-7 per pair of unit mass over the
cube of separations, the FP32 path by a constant, 5.2e-7.
The bound tells that the constant is there, not that the potentials are exact."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,seed", [(1000, 3), (2048, 11), (4096, 1)])
def test_mean_potential(n, seed, oracle_mod):
    import tigergrav_b200 as tg
    from tigergrav_b200 import ics
    x = ics.uniform(n, seed)
    with tg.GravitySolver(n, theta=0.7, leaf_max=64) as s:
        phi, _ = s.set_particles(x).solve_gravity().get_forces()
    o = oracle_mod.Oracle(theta=0.7, ewald=True, leaf_max=64).set_particles(x)
    o.build().multipoles().walk().evaluate()
    assert abs(np.mean(phi - o.forces()[0])) < 4e-7
