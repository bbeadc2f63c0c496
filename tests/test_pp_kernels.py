"""PP direct and the pair part of the Jacobian product at the edges of the CUDA
kernels' ranges: sink leaves of 1 to 64 particles (every cut into lanes and
copies), lists below and above the length where the kernel changes, lists
of a large part of the tree (shares, quarters of leaves), sources about half a box
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
    "wide_48": (lambda: _uniform(20000, 4), 0.7, 48, True, None),
    "wide_leaf7": (lambda: _uniform(6000, 5), 0.6, 7, True, None),
    "wide_free_soft": (lambda: _clumps(9000, 6), 0.6, 32, False, 2e-3),
    "short_24": (lambda: _uniform(20000, 4), 0.7, 24, True, None),
    "short_leaf7": (lambda: _uniform(6000, 5), 0.7, 7, True, None),
    "short_free_soft": (lambda: _clumps(12000, 6), 0.7, 16, False, 2e-3),
    "short_free_60": (lambda: _clumps(60000, 7), 0.8, 60, False, 1e-3),
    "long_leaf1": (lambda: _uniform(2000, 7), 0.25, 1, True, None),
    "long_leaf12": (lambda: _uniform(9000, 8), 0.25, 12, True, None),
    "long_leaf26": (lambda: _uniform(17000, 9), 0.25, 26, False, None),
    "long_clumps_58": (lambda: _clumps(40000, 10), 0.25, 58, False, 1e-3),
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


def test_jacobian_sums_keep_small_terms():
    """Two sources at +-1/16 of a sink, upstream gradients +-2^14, first in the order
    of the particles and in different copies of the sink: their terms (2^27 of unit
    mass) cancel to the bit, and the other pairs' terms stay, since every pair goes to
    a compensated sum of its copy: within 1e-5 of their sizes (their own rounding is a
    few 2^-24)."""
    import tigergrav_b200 as tg
    n = 64
    rng = np.random.default_rng(1)
    x = rng.integers(-2 ** 31, 2 ** 31, (n, 3)).astype(np.int32)
    x[4:, 0] &= 2 ** 31 - 1  # the upper half of the box: after the first four
    u = rng.standard_normal((n, 3))
    x[:4] = [[-2 ** 30, 0, 0], [-2 ** 30 + 2 ** 28, 0, 0], [-2 ** 30 - 2 ** 28, 0, 0], [-2 ** 30 + 2 ** 20, 0, 0]]
    u[:4] = [[0, 0, 0], [2.0 ** 14, 0, 0], [-2.0 ** 14, 0, 0], [0, 0, 0]]
    with tg.GravitySolver(n, theta=0.7, leaf_max=64, ewald=False, m=1.0 / n, soft_len=1e-3) as s:
        s.set_particles(x).build().multipoles().walk()
        got = s.tidal(u)[0]
        at = np.argsort(s.perm())  # sorted position of each particle; copy = position mod 2
    assert at[2] == 0 and at[1] == 3
    d = (x[0].astype(np.int64) - x[4:]) / 4294967296.0
    r = np.linalg.norm(d, axis=1)[:, None]
    t = -(-u[4:] / r ** 3 - 3.0 * d * (d * -u[4:]).sum(1)[:, None] / r ** 5) / n
    assert np.all(np.abs(got - t.sum(0)) <= 1e-5 * np.abs(t).sum(0))


def _seam(x, src, precision, ewald, h, kind="direct"):
    """(phi, g) of one sink group through the PP seam"""
    import torch
    from tigergrav_b200 import solver as tgs
    p = tgs.make_params(soft_len=h, m=1.0 / len(src), ewald=ewald, precision=precision)
    def off(n):
        return torch.tensor([0, n], dtype=torch.int64, device="cuda")
    f = torch.zeros((len(x), 4), dtype=torch.float64, device="cuda")
    tgs.gravity_PP(kind, p, off(len(x)), torch.from_numpy(x).cuda(), off(len(src)), torch.from_numpy(src).cuda(), f)
    return f.cpu().numpy()


@pytest.mark.parametrize("kind,ewald", [("direct", True), ("direct", False), ("ewald", True)])
@pytest.mark.parametrize("ns,ny", [(1, 1), (7, 128), (64, 1000), (130, 257)])
def test_seam_fp32_against_fp64(ns, ny, kind, ewald):
    """Sinks and sources up to a whole box apart (beyond the int32 range in free
    space), FP32 terms in FP64 sums: a term carries a few 2^-24, an Ewald term a few
    1e-7 of unit mass, so 2e-6 of the mean of the terms' sizes."""
    from tigergrav_b200 import ics
    rng = np.random.default_rng(ns + ny)
    x = ics.double_to_pos(np.concatenate([np.full((1, 3), 1e-9), rng.random((ns, 3))])[:ns])
    src = ics.double_to_pos(np.concatenate([np.full((1, 3), 1.0 - 1e-9), rng.random((ny, 3))])[:ny])
    a, b = (_seam(x, src, p, ewald, 1e-3, kind) for p in ("f32", "f64"))
    d = (x[:, None].astype(np.int64) - src[None].astype(np.int64)) / 4294967296.0
    if ewald:
        d -= np.round(d)
    r = np.maximum(np.sqrt((d ** 2).sum(-1)), 5e-4)
    size = 1.0 if kind == "ewald" else np.stack([(1 / r).mean(1)] + [(1 / r ** 2).mean(1)] * 3, 1)
    assert np.all(np.abs(a - b) <= 2e-6 * size)


def test_seam_infinite_term():
    """A term beyond FP32 (coincident particles, 1 / h past its range) is an
    infinite potential, not a NaN, and stays with its own sink."""
    x = np.array([[5, 6, 7], [2 ** 30, 0, 0]], np.int32)
    src = np.array([[2 ** 29, 1, 2], [5, 6, 7], [-2 ** 28, 8, 9]], np.int32)
    f = _seam(x, src, "f32", True, 6.5e-39)
    assert f[0, 0] == -np.inf and np.all(np.isfinite(f[1]))
