"""PP direct and the pair part of the Jacobian product at the edges of the CUDA
kernels' ranges: sink leaves of 1 to 64 particles (every cut into lanes and
copies), lists below and above the length where the kernel changes, fewer
leaves than SMs (list shares, quarters of leaves), sources about half a box
away (offsets beyond the int32 range), softened pairs."""
import numpy as np
import pytest

from helpers import arbiter_excess

pytestmark = pytest.mark.gpu


def _uniform(n, seed):
    return np.random.default_rng(seed).random((n, 3))


def _clumps(n, seed):
    """Half the particles in clumps of 1e-3 at the box's corner and centre: softened
    pairs, leaves of very different sizes, deep trees."""
    rng = np.random.default_rng(seed)
    x = rng.random((n, 3))
    k = n // 2
    x[:k] = (np.where(np.arange(k)[:, None] % 2, 0.5, 0.0) + 1e-3 * rng.standard_normal((k, 3))) % 1.0
    return x


CASES = {
    # name: (positions, theta, leaf_max, ewald, soft_len or None)
    "few_leaves_64": (lambda: _uniform(4096, 1), 0.7, 64, True, None),
    "few_leaves_one": (lambda: _uniform(61, 2), 0.7, 64, True, None),
    "few_free_33": (lambda: _uniform(1500, 3), 0.5, 33, False, None),
    "short_48": (lambda: _uniform(20000, 4), 0.7, 48, True, None),
    "short_leaf7": (lambda: _uniform(6000, 5), 0.6, 7, True, None),
    "short_free_soft": (lambda: _clumps(9000, 6), 0.6, 32, False, 2e-3),
    "long_leaf1": (lambda: _uniform(2000, 7), 0.3, 1, True, None),
    "long_leaf12": (lambda: _uniform(9000, 8), 0.3, 12, True, None),
    "long_leaf26": (lambda: _uniform(17000, 9), 0.3, 26, False, None),
    "long_clumps_58": (lambda: _clumps(40000, 10), 0.3, 58, False, 1e-3),
}


@pytest.mark.parametrize("name", list(CASES))
def test_pp_edges(name, oracle_mod):
    import tigergrav_b200 as tg
    from tigergrav_b200 import ics
    make, theta, leaf, ewald, h = CASES[name]
    x = ics.double_to_pos(make())
    kw = {} if h is None else dict(soft_len=h)
    with tg.GravitySolver(len(x), theta=theta, leaf_max=leaf, ewald=ewald, **kw) as s:
        s.set_particles(x).solve_gravity()
        phi, g = s.get_forces()
    o = oracle_mod.Oracle(theta=theta, ewald=ewald, leaf_max=leaf, **kw).set_particles(x)
    o.build().multipoles().walk().evaluate()
    rphi, rg = o.forces()
    o.evaluate(fp64=True)
    phi64, g64 = o.forces()
    fx, px = arbiter_excess(g, rg, g64, phi, rphi, phi64)
    assert fx <= 0.0 and px <= 0.0, (fx, px)


@pytest.mark.parametrize("n,theta,leaf,ewald", [(300, 0.7, 5, True), (70, 0.7, 64, True), (5000, 0.6, 64, True),
                                                (4000, 0.6, 48, False), (5000, 0.7, 128, True)])
def test_jacobian_fp32_against_fp64(n, theta, leaf, ewald):
    """J u in FP32 against the FP64 path on the same lists: FP32 pair Hessians carry
    ~1e-6 of their size, so 1e-5 of the rms product."""
    import tigergrav_b200 as tg
    from tigergrav_b200 import ics
    x = ics.double_to_pos(_uniform(n, 11))
    u = np.random.default_rng(12).standard_normal((n, 3))
    out = {}
    for p in ("f32", "f64"):
        with tg.GravitySolver(n, theta=theta, leaf_max=leaf, ewald=ewald, precision=p) as s:
            s.set_particles(x).build().multipoles().walk()
            out[p] = s.tidal(u)
    rms = np.sqrt(np.mean(out["f64"] ** 2))
    assert np.sqrt(np.mean((out["f32"] - out["f64"]) ** 2)) <= 1e-5 * rms
