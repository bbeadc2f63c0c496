"""One PP Ewald pair at a time: two particles of unit mass in a box, at a theta where
close ones are not a multipole either, with a softening so long (8) that the direct
force is below 0.03 and its rounding below 4e-9.  The FP32
path against the FP64 path over separations |x_d| <= lim, the bounds from the FP32
rounding of the outputs (|g| <= 1.5, |phi| <= 4: 4e-8 and 1e-7 rms) and of the mirror
images (at most 0.13 each; an erfc good to 1.5e-7 would add 1.2e-7 to the force)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SAMPLES = 200
LIMITS = (0.5, 0.25, 0.1, 0.05)


def _separations(lim):
    rng = np.random.default_rng(int(1000 * lim))
    a = rng.integers(-2 ** 31, 2 ** 31, (SAMPLES, 3))
    d = np.floor(rng.uniform(-lim, lim, (SAMPLES, 3)) * 2.0 ** 32).astype(np.int64)
    x = np.stack([a, a + d], 1)
    return ((x + 2 ** 31) % 2 ** 32 - 2 ** 31).astype(np.int32)


def _run(pairs, precision, call):
    import tigergrav_b200 as tg
    with tg.GravitySolver(2, theta=0.01, leaf_max=64, m=1.0, soft_len=8.0, precision=precision) as s:
        return [call(s.set_particles(x).solve_gravity()) for x in pairs]


@pytest.mark.parametrize("lim", LIMITS)
def test_force_and_potential(lim):
    x = _separations(lim)
    f32, f64 = (_run(x, p, lambda s: s.get_forces()) for p in ("f32", "f64"))
    dg = np.array([a[1] - b[1] for a, b in zip(f32, f64)])
    dphi = np.array([a[0] - b[0] for a, b in zip(f32, f64)])
    assert np.sqrt((dg ** 2).sum(-1).mean()) <= 2.5e-7
    # the mean that is kept on purpose, -5.2e-7
    assert abs(dphi.mean() + 5.0e-7) <= 1e-7
    assert dphi.std() <= 2e-7


@pytest.mark.parametrize("lim", LIMITS)
def test_jacobian(lim):
    """D2 (u_i - u_j) of ~10: FP32 rounding of the images' second derivatives, up to ~4."""
    x = _separations(lim)
    u = np.random.default_rng(3).standard_normal((2, 3))
    j32, j64 = (np.array(_run(x, p, lambda s: s.tidal(u))) for p in ("f32", "f64"))
    assert np.sqrt(((j32 - j64) ** 2).sum(-1).mean()) <= 2e-6


@pytest.mark.parametrize("precision", ["f32", "f64"])
@pytest.mark.parametrize("n,leaf", [(70, 64), (300, 20)])
def test_jacobian_of_a_translation(n, leaf, precision):
    """J depends on the differences of u alone.  Here every interaction is a pair
    (theta and softening), so a common u gives zero but for the FP64 rounding of
    the reciprocal sums, whose factors reach ~80 per unit u."""
    import tigergrav_b200 as tg
    from tigergrav_b200 import ics
    u = np.tile([1000.0, -300.0, 1.0 / 3.0], (n, 1))
    with tg.GravitySolver(n, theta=0.01, leaf_max=leaf, soft_len=8.0, precision=precision) as s:
        s.set_particles(ics.uniform(n, 3)).solve_gravity()
        c = s.stats()["counts"]
        assert c["CC_D"] == c["CC_E"] == c["PC_D"] == c["PC_E"] == c["CP_D"] == c["CP_E"] == 0
        assert np.abs(s.tidal(u)).max() <= 1e-11 * 1000.0
