"""The workloads that the framework's speed is measured on, through its public
entry points (tigergrav_b200.solver): whole force evaluations over the range
of box sizes, opening angles, leaf sizes and options that a simulation uses,
the leapfrog, the adjoint, batches of boxes, group finding, and two of the
kernel-level seams.

``listed()`` and ``draw(rng)`` give cases (plain dicts), ``prepare(case, seed)``
the handles and inputs a program holds before the call, ``run(state)`` one pass,
``work(case)`` what a pass cannot do without and ``exact(case, seed)`` the value
of the seams' outputs in 64 bits.  Inputs are made on the GPU from the seed:
a displaced lattice (P(k) ~ k^-2, rms displacement half the mean spacing, as
``ics.clustered``), i.i.d. uniform particles, or ``ics.halos``.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from tigergrav_b200 import ics
from tigergrav_b200 import solver as tgs

DEV = "cuda"


# ---------------------------------------------------------------- the cases

def listed():
    return [
        # the smallest evaluation: launches, host round trips and latency count
        dict(name="solve_4k_uniform", kind="solve", ic="uniform", n=4096, theta=0.7, leaf=64, ewald=True,
             precision="f32"),
        # the plain-method configuration: 32^3 uniform, theta 0.7, periodic
        dict(name="solve_32k_uniform", kind="solve", ic="uniform", n=32768, theta=0.7, leaf=64, ewald=True,
             precision="f32"),
        # an isolated system (no periodic images), odd particle count, concentrated haloes
        dict(name="solve_100k_free_halos", kind="solve", ic="halos", n=100003, theta=0.6, leaf=32, ewald=False,
             precision="f32"),
        # an odd lattice between the two regimes: moderate accuracy, small leaves
        dict(name="solve_101_theta05", kind="solve", ic="clustered", n=101 ** 3, theta=0.5, leaf=32, ewald=True,
             precision="f32"),
        # 128^3 at the opening angle that gives a force error of 1e-4 (production accuracy)
        dict(name="solve_128_theta02", kind="solve", ic="clustered", n=128 ** 3, theta=0.2, leaf=64, ewald=True,
             precision="f32"),
        # the largest box: 256^3 at a force error of 1e-4
        dict(name="solve_256_theta019", kind="solve", ic="clustered", n=256 ** 3, theta=0.19, leaf=48, ewald=True,
             precision="f32"),
        # the FP64 option: reference values, energy checks
        dict(name="solve_64_f64", kind="solve", ic="clustered", n=64 ** 3, theta=0.6, leaf=64, ewald=True,
             precision="f64"),
        # time integration: 128^3 clustered at theta 0.7, one evaluation and 10 kick-drift-kick steps
        dict(name="leapfrog_128_theta07", kind="leapfrog", ic="clustered", n=128 ** 3, theta=0.7, leaf=64, steps=10),
        # differentiation: forward steps with checkpoints and the adjoint pass back through them
        dict(name="adjoint_64_2steps", kind="adjoint", ic="clustered", n=64 ** 3, theta=0.7, leaf=64, steps=2),
        # 64 independent boxes of 2^12 to 2^18 particles in one call
        dict(name="batch_64_boxes", kind="batch", boxes=64, lo=12.0, hi=18.0, theta=0.7, leaf=64),
        # friends-of-friends groups at an output time: the group id of every particle
        dict(name="groups_262k", kind="groups", ic="halos", n=262144, link=0.2),
        # the kernel-level seams of a caller with its own lists: particle-particle, and node-node Ewald
        dict(name="seam_pp_direct", kind="seam_pp", groups=4096, sinks=64, sources=2048),
    ]


def draw(rng):
    kind = rng.choice(["solve"] * 6 + ["leapfrog", "adjoint", "batch", "groups", "seam_pp"])

    def log_int(a, b):
        return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))

    if kind == "solve":
        precision = "f64" if rng.random() < 0.15 else "f32"
        ic = rng.choice(["uniform", "clustered", "clustered", "halos"])
        n = log_int(2000, 100000 if precision == "f64" or ic == "halos" else 3000000)
        leaf = rng.choice([16, 32, 48, 64])
        if ic == "clustered":
            n = max(12, round(n ** (1.0 / 3.0))) ** 3
        # below this angle every leaf pair of a small box is an Ewald pair: nobody opens that far there
        lo = min(0.65, max(0.25, 8.0 * (leaf / n) ** (1.0 / 3.0)))
        return dict(kind="solve", ic=ic, n=n, theta=round(rng.uniform(lo, 0.8), 3), leaf=leaf,
                    ewald=rng.random() < 0.8, precision=precision)
    if kind in ("leapfrog", "adjoint"):
        n = max(16, round(log_int(5000, 1500000 if kind == "leapfrog" else 250000) ** (1.0 / 3.0))) ** 3
        return dict(kind=kind, ic="clustered", n=n, theta=round(rng.uniform(0.55, 0.8), 3),
                    leaf=rng.choice([32, 48, 64]), steps=rng.randint(2, 8) if kind == "leapfrog" else 2)
    if kind == "batch":
        return dict(kind="batch", boxes=rng.randint(5, 64), lo=12.0, hi=round(rng.uniform(14.0, 18.0), 2),
                    theta=round(rng.uniform(0.6, 0.8), 3), leaf=rng.choice([32, 64]))
    if kind == "groups":
        return dict(kind="groups", ic="halos", n=log_int(5000, 400000), link=round(rng.uniform(0.15, 0.25), 3))
    return dict(kind="seam_pp", groups=log_int(200, 5000), sinks=rng.randint(9, 100), sources=log_int(100, 2500))


# ---------------------------------------------------------------- inputs

def _generator(seed, salt=0):
    g = torch.Generator(device=DEV)
    g.manual_seed(1000003 * int(seed) + salt)
    return g


def _fixed(x):
    """Positions in [0, 1) to the 32-bit fixed point, x = i 2^-32 + 0.5."""
    z = torch.floor((x - 0.5) * 4294967296.0 + 0.5)
    return torch.where(z >= 2147483648.0, z - 4294967296.0, z).to(torch.int64).to(torch.int32).contiguous()


def _clustered(nside, seed, salt=0):
    """(positions, displacements) of the displaced lattice of ics.clustered, on the GPU."""
    f64 = torch.float64
    w = torch.randn((nside,) * 3, generator=_generator(seed, salt), device=DEV, dtype=f64)
    W = torch.fft.rfftn(w)
    k1 = 2.0 * math.pi * torch.fft.fftfreq(nside, d=1.0 / nside, device=DEV, dtype=f64)
    kz = 2.0 * math.pi * torch.fft.rfftfreq(nside, d=1.0 / nside, device=DEV, dtype=f64)
    kk = (k1[:, None, None], k1[None, :, None], kz[None, None, :])
    k2 = kk[0] ** 2 + kk[1] ** 2 + kk[2] ** 2
    k2[0, 0, 0] = 1.0
    amp = W / k2 ** 1.5
    amp[0, 0, 0] = 0.0
    psi = torch.stack([torch.fft.irfftn(1j * k * amp, s=(nside,) * 3) for k in kk], dim=-1).reshape(-1, 3)
    psi *= (0.5 / nside) / torch.sqrt((psi ** 2).sum(1).mean())
    g = torch.arange(nside, device=DEV, dtype=f64) / nside
    lat = torch.stack(torch.meshgrid(g, g, g, indexing="ij"), dim=-1).reshape(-1, 3)
    x = torch.remainder(lat + psi, 1.0)
    return torch.where(x >= 1.0, torch.zeros_like(x), x), psi


def _particles(ic, n, seed, salt=0):
    """(fixed-point positions, float32 velocities) on the GPU."""
    if ic == "clustered":
        x, psi = _clustered(round(n ** (1.0 / 3.0)), seed, salt)
        return _fixed(x), (3.0 * psi).float().contiguous()  # growing-mode flow
    if ic == "halos":
        x = torch.from_numpy(ics.halos(n, (1000003 * int(seed) + salt) % (1 << 31))).to(DEV)
    else:
        x = _fixed(torch.rand((n, 3), generator=_generator(seed, salt), device=DEV, dtype=torch.float64))
    v = 0.01 * torch.randn((n, 3), generator=_generator(seed, salt + 1), device=DEV, dtype=torch.float32)
    return x, v


def _group_offsets(total, mean, seed, salt):
    """Ragged CSR offsets: sizes spread evenly over [mean/2, 3 mean/2] (at least 1) in random order."""
    size = max(1, mean // 2) + torch.arange(total, device=DEV) % (mean + 1)
    size = size[torch.randperm(total, generator=_generator(seed, salt), device=DEV)]
    off = torch.zeros(total + 1, dtype=torch.int64, device=DEV)
    off[1:] = torch.cumsum(size, 0)
    return off


def _owner(off):
    return torch.repeat_interleave(torch.arange(len(off) - 1, device=DEV), off[1:] - off[:-1])


def _seam_pp_inputs(case, seed):
    """Sink groups of the size of a leaf with sources within three leaf widths, as the near lists of a 128^3 box."""
    ng = case["groups"]
    sink_off = _group_offsets(ng, case["sinks"], seed, 11)
    src_off = _group_offsets(ng, case["sources"], seed, 12)
    g = _generator(seed, 13)
    width = (64.0 / 128 ** 3) ** (1.0 / 3.0)
    c = torch.rand((ng, 3), generator=g, device=DEV, dtype=torch.float64)

    def around(off, w):
        u = torch.rand((int(off[-1]), 3), generator=g, device=DEV, dtype=torch.float64) - 0.5
        return _fixed(torch.remainder(c[_owner(off)] + w * u, 1.0))

    return sink_off, around(sink_off, width), src_off, around(src_off, 3.0 * width)


# ---------------------------------------------------------------- one pass

def prepare(case, seed):
    kind = case["kind"]
    if kind == "seam_pp":
        sink_off, sink_x, src_off, src_x = _seam_pp_inputs(case, seed)
        p = tgs.make_params(n=128 ** 3)
        f = torch.zeros((len(sink_x), 4), dtype=torch.float64, device=DEV)
        return dict(kind=kind, p=p, sink_off=sink_off, sink_x=sink_x, src_off=src_off, src_x=src_x, f=f)
    if kind == "batch":
        counts = ics.batch_sizes(case["boxes"], 4, case["lo"], case["hi"])
        xs = []
        for b, n in enumerate(counts):  # even boxes uniform, odd ones clustered on the nearest cube
            if b % 2 == 0:
                xs.append(_particles("uniform", int(n), seed, 10 * b)[0])
            else:
                xs.append(_particles("clustered", max(2, round(float(n) ** (1.0 / 3.0))) ** 3, seed, 10 * b)[0])
        counts = np.array([len(x) for x in xs], np.int64)
        h = tgs.GravityBatch(counts, theta=case["theta"], leaf_max=case["leaf"])
        return dict(kind=kind, h=h, x=torch.cat(xs).cpu().numpy())
    x, v = _particles(case["ic"], case["n"], seed)
    n = len(x)
    s = dict(kind=kind, x=x, v=v)
    if kind == "groups":
        s["h"], s["link"] = tgs.GravitySolver(n), case["link"]
        return s
    f64 = case.get("precision", "f32") == "f64"
    s["h"] = tgs.GravitySolver(n, theta=case["theta"], leaf_max=case["leaf"], ewald=case.get("ewald", True),
                               precision="f64" if f64 else "f32")
    if kind == "solve":
        dt = torch.float64 if f64 else torch.float32
        s["phi"] = torch.empty(n, dtype=dt, device=DEV)
        s["g"] = torch.empty((n, 3), dtype=dt, device=DEV)
    else:
        s["steps"] = case["steps"]
    if kind == "adjoint":
        s["w"] = torch.randn((n, 3), generator=_generator(seed, 5), device=DEV, dtype=torch.float64).cpu().numpy()
    return s


def run(state):
    kind = state["kind"]
    if kind == "seam_pp":
        state["f"].zero_()  # the seams add to f
        tgs.gravity_PP("direct", state["p"], state["sink_off"], state["sink_x"], state["src_off"], state["src_x"],
                       state["f"])
        return state["f"]
    h = state["h"]
    if kind == "batch":
        phi, g = h.set_particles(state["x"]).solve().get_forces()
        return phi, g
    if kind == "solve":
        h.set_particles(state["x"]).solve_gravity()
        h.get_forces(out_phi=state["phi"], out_g=state["g"])
        return state["phi"], state["g"]
    h.set_particles(state["x"], state["v"])
    if kind == "groups":
        return h.find_groups(state["link"])
    if kind == "leapfrog":
        h.leapfrog(1.0e-3, state["steps"])
        x, v = h.get_particles()
        return ics.pos_to_double(x), v
    gx0, gv0 = h.forward(1.0e-3, state["steps"]).backward(state["w"])
    return gx0, gv0


# ---------------------------------------------------------------- the floor

def _solve_work(n, theta, leaf, ewald, precision):
    """One evaluation: particles in, forces out; the particle pairs that the
    opening angle leaves to direct summation (leaves within (r_a + r_b)/theta,
    with radii of 0.8 leaf widths at 0.6 leaf_max particles) at 18 operations,
    the node pairs of the far field (one per 0.05 pair at 1025), and with the
    periodic correction one smooth contraction per 4 of those."""
    pairs = n * min(float(n), 17.0 * 0.6 * leaf / theta ** 3)
    nodes = 0.05 * pairs / (0.6 * leaf)
    flops = 18.0 * pairs + 1025.0 * nodes * (1.25 if ewald else 1.0)
    return dict(bytes=n * (12.0 + 16.0 * (2 if precision == "f64" else 1)), flops=flops)


def work(case):
    kind = case["kind"]
    if kind == "seam_pp":
        pairs = float(case["groups"]) * case["sinks"] * case["sources"]
        return dict(bytes=case["groups"] * (44.0 * case["sinks"] + 12.0 * case["sources"]), flops=18.0 * pairs)
    if kind == "batch":
        ws = [_solve_work(float(n), case["theta"], case["leaf"], True, "f32")
              for n in ics.batch_sizes(case["boxes"], 4, case["lo"], case["hi"])]
        return dict(bytes=sum(w["bytes"] for w in ws), flops=sum(w["flops"] for w in ws))
    n = case["n"]
    if kind == "groups":  # positions and velocities in, 64-bit ids out; a few pair tests per particle
        return dict(bytes=32.0 * n, flops=60.0 * 8 * n)
    w = _solve_work(n, case["theta"], case["leaf"], case.get("ewald", True), case.get("precision", "f32"))
    if kind == "leapfrog":
        return dict(bytes=48.0 * n, flops=w["flops"] * (1 + case["steps"]))
    if kind == "adjoint":  # K + 1 evaluations forward, K Jacobian products of twice the pair work back
        return dict(bytes=(24.0 + 72.0) * n, flops=w["flops"] * (1 + 3 * case["steps"]))
    return w


# ---------------------------------------------------------------- 64 bits

def exact(case, seed):
    """The seam's sums in 64 bits.  A tree evaluation has no such value: its
    result is defined by the interaction lists, whose opening error is far
    above rounding, so it is held against earlier results alone."""
    if case["kind"] != "seam_pp":
        return None
    sink_off, sink_x, src_off, src_x = _seam_pp_inputs(case, seed)
    n = 128 ** 3
    h, m = 0.02 * n ** (-1.0 / 3.0), 1.0 / n
    f = torch.zeros((len(sink_x), 4), dtype=torch.float64, device=DEV)
    so, yo = sink_off.tolist(), src_off.tolist()
    step = max(1, 20_000_000 // (2 * case["sinks"] * case["sources"]))
    for g0 in range(0, len(so) - 1, step):  # a few groups at a time, padded to their largest
        g1 = min(len(so) - 1, g0 + step)
        ns = max(so[g + 1] - so[g] for g in range(g0, g1))
        ny = max(yo[g + 1] - yo[g] for g in range(g0, g1))
        a, b = sink_off[g0:g1, None] + torch.arange(ns, device=DEV), src_off[g0:g1, None] + torch.arange(ny, device=DEV)
        ma, mb = a < sink_off[g0 + 1:g1 + 1, None], b < src_off[g0 + 1:g1 + 1, None]
        X, Y = sink_x[a.clamp(max=len(sink_x) - 1)], src_x[b.clamp(max=len(src_x) - 1)]
        d = X[:, :, None, :].to(torch.int64) - Y[:, None, :, :].to(torch.int64)
        d = (torch.remainder(d + 2147483648, 4294967296) - 2147483648).double() / 4294967296.0  # nearest image
        r = torch.sqrt((d * d).sum(-1))
        u = torch.clamp(r / h, max=1.0)
        us = torch.clamp(u, min=0.5)
        fi = 32.0 / 3.0 - 38.4 * u ** 2 + 32.0 * u ** 3  # the spline softening, inner and outer half
        fo = 64.0 / 3.0 - 48.0 * us + 38.4 * us ** 2 - 32.0 / 3.0 * us ** 3 - 1.0 / (15.0 * us ** 3)
        pi_ = 14.0 / 5.0 - 16.0 / 3.0 * u ** 2 + 48.0 / 5.0 * u ** 4 - 32.0 / 5.0 * u ** 5
        po = (-1.0 / (15.0 * us) + 16.0 / 5.0 - 32.0 / 3.0 * us ** 2 + 16.0 * us ** 3 - 48.0 / 5.0 * us ** 4
              + 32.0 / 15.0 * us ** 5)
        rs = torch.clamp(r, min=h)
        soft, inner = r <= h, u < 0.5
        F = torch.where(soft, torch.where(inner, fi, fo) / h ** 3, rs ** -3) * mb[:, None, :]
        P = torch.where(soft, torch.where(inner, pi_, po) / h, 1.0 / rs) * mb[:, None, :]
        out = torch.cat([-m * P.sum(-1, keepdim=True) + 315.0 / 128.0 * m / h, -m * (F[..., None] * d).sum(2)], -1)
        f[a[ma]] = out[ma]
    return f
