"""Performance cases: the calls that programs built on this library make, from
a ten-thousand-particle differentiable step to million-particle walks, each
through a public entry point of ``sbh_b200``.

``listed()`` names twelve of them and ``draw()`` makes more over the same
ranges. A case is a dict of plain values; its ``kind`` selects the entry point:

* ``gravity_step``     differentiable self-gravity (forward and backward, the
                       tree rebuilt in each) of one small or medium system
* ``gravity_force``    tree build + force of one system (an integrator's step)
* ``gravity_adjoint``  tree build + fused force and full adjoint of one system
* ``forest_adjoint``   the same for many independent systems in one forest
* ``treepm``           the periodic short-range half of a TreePM step
* ``winding``          winding number of an oriented surface sample
* ``winding_adjoint``  the same with its gradients
* ``octree8_step``     the reference-compatible octree8 step with its
                       recompute VJP
* ``direct_step``      the reference-compatible direct sum with its VJP
* ``mlpcv_step``       the reference-compatible stochastic octree8 estimate
                       and its VJP on a tree that the program holds
* ``stochastic_step``  native stochastic estimate and its adjoint
"""
from __future__ import annotations

import math
import os
import sys

import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "barnes-hut_b200"))

import sbh_b200 as B  # noqa: E402

DEV = "cuda"


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # The smallest benchmark configuration: 10,000 particles in the unit
        # cube, leaf size 8, differentiated with respect to positions and
        # masses. A fit or a training loop calls this thousands of times.
        dict(name="gravity_step_10k", kind="gravity_step", n=10000, dist="uniform", beta=2.0, softening=1e-3,
             leaf_size=8),
        # The plain force evaluation of a clustered million-particle system.
        dict(name="gravity_force_1m", kind="gravity_force", n=1 << 20, dist="plummer", beta=2.0, softening=1e-3,
             leaf_size=16, group_size=0),
        # The headline workload's unit: force and full adjoint of 2^20 particles.
        dict(name="gravity_adjoint_1m", kind="gravity_adjoint", n=1 << 20, dist="plummer", beta=2.0, softening=1e-3,
             leaf_size=16, group_size=0),
        # A batch of independent systems of very uneven sizes in one forest.
        dict(name="forest_adjoint_40", kind="forest_adjoint", systems=40, n_lo=1000, n_hi=200000, beta=2.0,
             softening=1e-3, leaf_size=16),
        # The short-range half of a TreePM step on 128^3 lattice particles.
        dict(name="treepm_force_2m", kind="treepm", cells=128, r_split=1.0, prune=4.0, softening=0.1, beta=1.7,
             group_size=64, adjoint=False),
        # Inside/outside field of an ellipsoid sample on a million points.
        dict(name="winding_1m", kind="winding", n=262144, m=1 << 20, beta=2.0, leaf_size=16),
        # Gradients of the winding number for shape fitting, ragged sizes.
        dict(name="winding_adjoint_200k", kind="winding_adjoint", n=60001, m=200003, beta=2.0, leaf_size=16),
        # The reference-compatible octree8 step at its defaults, a small system.
        dict(name="octree8_step_5k", kind="octree8_step", n=5000, dist="uniform", depth=5, beta=2.0, softening=1e-2,
             cutoff=1.0, prune=True),
        # The same on a clustered system without a cutoff (plain gravity).
        dict(name="octree8_step_256k", kind="octree8_step", n=1 << 18, dist="plummer", depth=7, beta=2.0,
             softening=1e-3, cutoff=1e7, prune=False),
        # Direct summation at the reference's defaults, the size of its demos.
        dict(name="direct_step_4k", kind="direct_step", n=4096, dist="uniform", softening=1e-2, cutoff=1.0,
             periodic=False),
        # The reference's stochastic estimator on a held octree8.
        dict(name="mlpcv_step_100k", kind="mlpcv_step", n=100003, m=65536, depth=6, beta=1.0, samples=1,
             softening=1e-3, cutoff=1e7),
        # The native stochastic estimate, 32 nodes per query, and its adjoint.
        dict(name="stochastic_step_500k", kind="stochastic_step", n=1 << 19, dist="plummer", beta=2.0,
             beta_coarse=1.0, samples=32, softening=1e-3, leaf_size=16),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["gravity_step", "gravity_force", "gravity_adjoint", "forest_adjoint", "treepm", "winding",
                       "winding_adjoint", "octree8_step", "direct_step", "mlpcv_step", "stochastic_step"])
    if kind == "gravity_step":
        return dict(kind=kind, n=_log_int(rng, 1000, 200000), dist=rng.choice(["uniform", "plummer"]),
                    beta=rng.choice([2.0, 1.0 / 0.6]), softening=rng.choice([1e-3, 2e-3]),
                    leaf_size=rng.choice([8, 16, 24]))
    if kind in ("gravity_force", "gravity_adjoint"):
        dist = rng.choice(["uniform", "plummer", "lattice"])
        return dict(kind=kind, n=_log_int(rng, 2000, 1 << 20), dist=dist,
                    beta=1.0 / 0.6 if dist == "lattice" else 2.0, softening=2e-3 if dist == "lattice" else 1e-3,
                    leaf_size=16, group_size=rng.choice([0, 64, 96]))
    if kind == "forest_adjoint":
        return dict(kind=kind, systems=rng.randint(4, 40), n_lo=1000, n_hi=_log_int(rng, 2000, 200000), beta=2.0,
                    softening=1e-3, leaf_size=16)
    if kind == "treepm":
        adjoint = rng.random() < 0.5
        return dict(kind=kind, cells=rng.randint(24, 96 if adjoint else 128), r_split=1.0, prune=4.0, softening=0.1,
                    beta=1.7, group_size=rng.choice([32, 64, 96]), adjoint=adjoint)
    if kind == "winding":
        return dict(kind=kind, n=_log_int(rng, 5000, 262144), m=_log_int(rng, 5000, 1 << 20), beta=2.0, leaf_size=16)
    if kind == "winding_adjoint":
        return dict(kind=kind, n=_log_int(rng, 5000, 200000), m=_log_int(rng, 5000, 400000), beta=2.0, leaf_size=16)
    if kind == "octree8_step":
        unit = rng.random() < 0.5
        n = _log_int(rng, 1000, 60000 if unit else 1 << 18)
        return dict(kind=kind, n=n, dist="uniform" if unit else "plummer",
                    depth=5 if n < 20000 else (6 if unit else 7), beta=2.0, softening=1e-2 if unit else 1e-3,
                    cutoff=1.0 if unit else 1e7, prune=unit)
    if kind == "direct_step":
        unit = rng.random() < 0.6
        return dict(kind=kind, n=_log_int(rng, 500, 60000), dist="uniform" if unit else "plummer",
                    softening=1e-2 if unit else 1e-3, cutoff=rng.choice([0.2, 1.0]) if unit else 1e7,
                    periodic=unit and rng.random() < 0.4)
    if kind == "mlpcv_step":
        return dict(kind=kind, n=_log_int(rng, 10000, 200000), m=_log_int(rng, 2000, 65536),
                    depth=rng.choice([5, 6]), beta=1.0, samples=rng.choice([1, 2]), softening=1e-3, cutoff=1e7)
    return dict(kind="stochastic_step", n=_log_int(rng, 20000, 1 << 19), dist=rng.choice(["uniform", "plummer"]),
                beta=2.0, beta_coarse=rng.choice([1.0, 1.25, 1.5]), samples=rng.choice([16, 32]), softening=1e-3,
                leaf_size=16)


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed) * 2654435761 % (1 << 62))


def _rand(g, *shape):
    return torch.rand(*shape, generator=g, device=DEV, dtype=torch.float64)


def _normal(g, *shape):
    return torch.randn(*shape, generator=g, device=DEV, dtype=torch.float64)


def _plummer(g, n):
    """Plummer sphere of scale radius 1 truncated at radius 10 (exact inverse CDF)."""
    m_max = 1000.0 / 101.0 ** 1.5
    x = (_rand(g, n) * m_max).clamp_min(1e-300)
    r = (x ** (-2.0 / 3.0) - 1.0).rsqrt()
    c = 2.0 * _rand(g, n) - 1.0
    phi = 2.0 * math.pi * _rand(g, n)
    s = (1.0 - c * c).sqrt()
    return torch.stack([r * s * phi.cos(), r * s * phi.sin(), r * c], 1).float()


def _lattice(g, k):
    """k^3 lattice of unit spacing, each point displaced by 0.2 cells rms."""
    a = torch.arange(k, device=DEV, dtype=torch.float64) + 0.5
    p = torch.stack(torch.meshgrid(a, a, a, indexing="ij"), -1).reshape(-1, 3)
    return p + _normal(g, k ** 3, 3) * (0.2 / math.sqrt(3.0))


def _points(g, dist, n):
    if dist == "plummer":
        return _plummer(g, n)
    if dist == "uniform":
        return _rand(g, n, 3).float()
    k = max(2, math.ceil(n ** (1.0 / 3.0) - 1e-9))
    p = _lattice(g, k) / k
    return p[torch.randperm(k ** 3, generator=g, device=DEV)[:n]].float().contiguous()


def _ellipsoid(g, n, axes=(1.0, 0.7, 0.5)):
    """Oriented samples of an ellipsoid: directions from a normal deviate,
    outward unit normals, weights proportional to the area each stands for."""
    ax = torch.tensor(axes, device=DEV, dtype=torch.float64)
    v = _normal(g, n, 3)
    v = v / v.norm(dim=1, keepdim=True)
    p = v * ax
    nrm = v / ax
    area = nrm.norm(dim=1) * ax.prod() * (4.0 * math.pi / n)
    nrm = nrm / nrm.norm(dim=1, keepdim=True)
    return p.float(), nrm.float(), area.float()


def prepare(case, seed):
    g = _gen(seed)
    kind = case["kind"]
    s = dict(case=case)
    if kind in ("gravity_step", "gravity_force", "gravity_adjoint", "stochastic_step", "octree8_step", "direct_step"):
        n = case["n"]
        s["x"] = _points(g, case["dist"], n)
        s["m"] = torch.full((n,), 1.0 / n, device=DEV)
        s["w"] = _normal(g, n, 3).float()
        s["seed"] = int(seed) % 1000003
    elif kind == "forest_adjoint":
        lo, hi = math.log(case["n_lo"]), math.log(case["n_hi"])
        # the sizes are the batch's shape, the same for every seed
        f = [((i + 1) * 0.6180339887498949) % 1.0 for i in range(case["systems"])]
        sizes = [int(math.exp(lo + (hi - lo) * u)) for u in f]
        offs = [0]
        for k in sizes:
            offs.append(offs[-1] + k)
        s["x"] = _plummer(g, offs[-1])
        s["m"] = torch.cat([torch.full((k,), 1.0 / k, device=DEV) for k in sizes])
        s["w"] = _normal(g, offs[-1], 3).float()
        s["offsets"] = torch.tensor(offs, dtype=torch.int64, device=DEV)
        s["sizes"] = sizes
    elif kind == "treepm":
        k = case["cells"]
        s["x"] = torch.remainder(_lattice(g, k), float(k)).float().clamp_max(k * (1.0 - 1e-7))
        s["m"] = torch.ones(k ** 3, device=DEV)
        s["w"] = _normal(g, k ** 3, 3).float()
    elif kind in ("winding", "winding_adjoint"):
        s["x"], s["nrm"], s["m"] = _ellipsoid(g, case["n"])
        s["q"] = (3.0 * _rand(g, case["m"], 3) - 1.5).float()
        s["u"] = _normal(g, case["m"]).float()
    else:  # mlpcv_step
        s["x"] = _plummer(g, case["n"])
        s["m"] = torch.full((case["n"],), 1.0 / case["n"], device=DEV)
        s["leaf"], s["node"] = B.build_octree8_buffers(s["x"], torch.zeros_like(s["x"]), s["m"],
                                                       max_depth=case["depth"])
        s["q"] = _plummer(g, case["m"])
        s["w"] = _normal(g, case["m"], 3).float()
        s["seed"] = int(seed) % 1000003
    if kind in ("gravity_force", "gravity_adjoint", "forest_adjoint", "treepm", "winding"):
        s["tree"] = B.NativeTree()  # the handle an integrator or a field evaluator keeps
    return s


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def run(state):
    s, c = state, state["case"]
    kind = c["kind"]
    if kind == "gravity_step":
        x, m = s["x"].detach().requires_grad_(), s["m"].detach().requires_grad_()
        a = B.native_force_recompute_vjp(x, m, beta=c["beta"], softening=c["softening"], leaf_size=c["leaf_size"])
        gx, gm = torch.autograd.grad(a, (x, m), s["w"])
        return a.detach(), gx, gm
    if kind in ("gravity_force", "gravity_adjoint"):
        adj = kind == "gravity_adjoint"
        s["tree"].build(s["x"], s["m"], leaf_size=c["leaf_size"], with_adjoint=adj,
                        group_size=c["group_size"] or None)
        if not adj:
            return s["tree"].force(beta=c["beta"], softening=c["softening"])
        return s["tree"].force_vjp(s["w"], beta=c["beta"], softening=c["softening"])
    if kind == "forest_adjoint":
        s["tree"].build(s["x"], s["m"], None, s["offsets"], leaf_size=c["leaf_size"])
        return s["tree"].force_vjp(s["w"], beta=c["beta"], softening=c["softening"])
    if kind == "treepm":
        kw = dict(beta=c["beta"], softening=c["softening"], cutoff=c["r_split"], quadrupole=False, periodic=True,
                  box_length=float(c["cells"]), prune_radius=c["prune"] * c["r_split"])
        s["tree"].build(s["x"], s["m"], with_adjoint=c["adjoint"], group_size=c["group_size"])
        return s["tree"].force_vjp(s["w"], **kw) if c["adjoint"] else s["tree"].force(**kw)
    if kind == "winding":
        s["tree"].build(s["x"], s["m"], normals=s["nrm"], leaf_size=c["leaf_size"], with_adjoint=False)
        return s["tree"].winding_number(s["q"], beta=c["beta"])
    if kind == "winding_adjoint":
        ins = [s[k].detach().requires_grad_() for k in ("x", "nrm", "m", "q")]
        w = B.native_winding_number(*ins, beta=c["beta"], leaf_size=c["leaf_size"])
        return (w.detach(),) + torch.autograd.grad(w, ins, s["u"])
    if kind == "octree8_step":
        x, m = s["x"].detach().requires_grad_(), s["m"].detach().requires_grad_()
        a = B.softened_barnes_hut_force_octree8_recompute_vjp(
            x, m, beta=c["beta"], softening_scale=c["softening"], cutoff_scale=c["cutoff"], max_depth=c["depth"],
            prune_enabled=c["prune"])
        gx, gm = torch.autograd.grad(a, (x, m), s["w"])
        return a.detach(), gx, gm
    if kind == "direct_step":
        x, m = s["x"].detach().requires_grad_(), s["m"].detach().requires_grad_()
        a = B.softened_direct_force_recompute_vjp(x, m, softening_scale=c["softening"], cutoff_scale=c["cutoff"],
                                                  periodic=c["periodic"], box_length=1.0)
        gx, gm = torch.autograd.grad(a, (x, m), s["w"])
        return a.detach(), gx, gm
    if kind == "mlpcv_step":
        kw = dict(beta=c["beta"], samples_per_subdomain=c["samples"], seed=s["seed"], softening_scale=c["softening"],
                  cutoff_scale=c["cutoff"], prune_enabled=False)
        f = B.softened_stochastic_barnes_hut_force_octree8(s["leaf"], s["node"], s["q"], **kw)
        return f, B.softened_stochastic_barnes_hut_force_octree8_vjp(s["leaf"], s["node"], s["q"], s["w"], **kw)
    x, m = s["x"].detach().requires_grad_(), s["m"].detach().requires_grad_()
    a = B.native_stochastic_force(x, m, beta=c["beta"], beta_coarse=c["beta_coarse"], samples=c["samples"],
                                  seed=s["seed"], softening=c["softening"], leaf_size=c["leaf_size"])
    gx, gm = torch.autograd.grad(a, (x, m), s["w"])
    return a.detach(), gx, gm


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def _interactions(n, beta):
    """Tree interactions per query at opening beta: about 12,300 at 2^20 and
    beta 2 (the reference's opening rule on a Plummer sphere), one more shell
    of about 1,000 per doubling, the volume of a shell going with beta^2.6."""
    return min(float(n), 1000.0 * max(1.0, math.log2(max(n, 2)) - 7.7) * (beta / 2.0) ** 2.6)


def work(case):
    """Bytes: inputs read once, outputs written once. Flops: 20 per pair or
    accepted node for a force (15 for a winding number), 60 with its VJP."""
    c = case
    kind = c["kind"]
    if kind == "forest_adjoint":
        lo, hi = math.log(c["n_lo"]), math.log(c["n_hi"])
        sizes = [int(math.exp(lo + (hi - lo) * (((i + 1) * 0.6180339887498949) % 1.0))) for i in range(c["systems"])]
        return dict(bytes=56.0 * sum(sizes), flops=sum(60.0 * k * _interactions(k, c["beta"]) for k in sizes))
    if kind == "treepm":
        n = c["cells"] ** 3
        pairs = 4.0 / 3.0 * math.pi * (c["prune"] * c["r_split"]) ** 3
        return dict(bytes=(56.0 if c["adjoint"] else 28.0) * n, flops=(60.0 if c["adjoint"] else 20.0) * n * pairs)
    if kind in ("winding", "winding_adjoint"):
        i = 0.25 * _interactions(c["n"], c["beta"])
        if kind == "winding":
            return dict(bytes=28.0 * c["n"] + 16.0 * c["m"], flops=15.0 * c["m"] * i)
        return dict(bytes=56.0 * c["n"] + 32.0 * c["m"], flops=45.0 * c["m"] * i)
    n = float(c["n"])
    if kind == "direct_step":
        return dict(bytes=56.0 * n, flops=60.0 * n * n)
    if kind == "mlpcv_step":
        return dict(bytes=16.0 * n + 48.0 * c["m"], flops=60.0 * c["m"] * 300.0 * (1.0 + 3.0 * c["samples"]))
    if kind == "stochastic_step":
        return dict(bytes=56.0 * n, flops=60.0 * n * _interactions(n, c["beta_coarse"]))
    if kind == "gravity_force":
        return dict(bytes=28.0 * n, flops=20.0 * n * _interactions(n, c["beta"]))
    return dict(bytes=56.0 * n, flops=60.0 * n * _interactions(n, c["beta"]))


def tolerance(case):
    """FP32 sums of up to some ten thousand terms in another order, the plan
    (tree, groups, opening decisions, sampled paths) being the same."""
    kind = case["kind"]
    if kind == "mlpcv_step":
        # a sampled path whose probability ties with its draw may turn
        return dict(rel=1e-4, max=2e-2)
    if kind == "direct_step":
        return dict(rel=2e-6, max=2e-4)  # 1e-7 and 3e-7 off the 64-bit sums
    return dict(rel=1e-5, max=1e-3)


# ---------------------------------------------------------------------------
# the same in 64 bits: direct sums over every pair
# ---------------------------------------------------------------------------
MOST_PAIRS = 1e11


def _chunks(m, n):
    step = max(1, (1 << 25) // max(n, 1))
    for a in range(0, m, step):
        yield a, min(m, a + step)


def _pair_terms(r2, eps2, cutoff):
    """s and t of the pair force s d (d = source - query): s = att h^(-3/2)
    with h = r^2 + eps^2, and t = (1 / r) ds/dr."""
    ih = 1.0 / (r2 + eps2)
    ih3 = ih * ih.sqrt()
    if not cutoff:
        return ih3, -3.0 * ih3 * ih
    r = (r2 + 1e-12).sqrt()
    u = r / (2.0 * cutoff)
    e = torch.exp(-u * u)
    att = torch.special.erfc(u) + (2.0 / math.sqrt(math.pi)) * u * e
    s = att * ih3
    return s, -3.0 * s * ih - ih3 * r * e / (2.0 * math.sqrt(math.pi) * cutoff ** 3)


def _gravity(x, m, w, eps2, cutoff=0.0, box=0.0, adjoint="full"):
    """(a, gx, gm) of sum w . a; adjoint: "none", "query" (the query-side
    gradient, gm zero) or "full"."""
    x, m = x.double(), m.double()
    w = w.double() if adjoint != "none" else None
    n = x.shape[0]
    a, gx, gm = torch.empty_like(x), torch.empty_like(x), torch.zeros_like(m)
    for lo, hi in _chunks(n, n):
        d = [x[None, :, k] - x[lo:hi, None, k] for k in range(3)]
        if box:
            d = [v - box * torch.round(v / box) for v in d]
        s, t = _pair_terms(d[0] * d[0] + d[1] * d[1] + d[2] * d[2], eps2, cutoff)
        ms = s * m
        for k in range(3):
            a[lo:hi, k] = (ms * d[k]).sum(1)
        if adjoint == "none":
            continue
        wk = w[lo:hi]
        # query side: -sum_j m_j (s w + t (d . w) d)
        mt = t * m * (d[0] * wk[:, :1] + d[1] * wk[:, 1:2] + d[2] * wk[:, 2:])
        for k in range(3):
            gx[lo:hi, k] = -ms.sum(1) * wk[:, k] - (mt * d[k]).sum(1)
        if adjoint == "full":  # source side, the pairs read the other way
            dw = d[0] * w[None, :, 0] + d[1] * w[None, :, 1] + d[2] * w[None, :, 2]
            gm[lo:hi] = -(dw * s).sum(1)
            dw = dw * t
            for k in range(3):
                gx[lo:hi, k] += m[lo:hi] * ((s * w[None, :, k]).sum(1) + (dw * d[k]).sum(1))
    return a, gx, gm


def _winding(x, nrm, m, q, u):
    """w, dL/dx, dL/dnrm, dL/dm, dL/dq of L = sum u w."""
    x, nrm, m, q, u = (v.double() for v in (x, nrm, m, q, u))
    k4 = 1.0 / (4.0 * math.pi)
    w, gq = torch.empty_like(u), torch.empty_like(q)
    gx, gn, gm = torch.zeros_like(x), torch.zeros_like(nrm), torch.zeros_like(m)
    for lo, hi in _chunks(q.shape[0], x.shape[0]):
        d = [x[None, :, k] - q[lo:hi, None, k] for k in range(3)]
        r = (d[0] * d[0] + d[1] * d[1] + d[2] * d[2]).sqrt()
        K = k4 / (r * r * r + 1e-5)
        nd = d[0] * nrm[:, 0] + d[1] * nrm[:, 1] + d[2] * nrm[:, 2]
        w[lo:hi] = (nd * K) @ m
        c = 3.0 * nd * r * K * K / k4
        uu = u[lo:hi]
        gm += uu @ (nd * K)
        for k in range(3):
            f = K * nrm[:, k] - c * d[k]
            gq[lo:hi, k] = -uu * (f @ m)
            gx[:, k] += m * (uu @ f)
            gn[:, k] += m * (uu @ (d[k] * K))
    return w, gx, gn, gm, gq


def exact(case, seed):
    c = case
    kind = c["kind"]
    if kind == "mlpcv_step":
        return None  # an estimate from sampled paths
    n = c["cells"] ** 3 if kind == "treepm" else c.get("n", 0)
    pairs = float(n) * (c["m"] if kind.startswith("winding") else n)
    if kind == "forest_adjoint":
        pairs = c["systems"] * 0.25 * float(c["n_hi"]) ** 2
    if kind == "treepm":
        pairs *= 3.0
    if pairs > MOST_PAIRS:
        return None
    s = prepare(case, seed)
    if kind.startswith("winding"):
        w, gx, gn, gm, gq = _winding(s["x"], s["nrm"], s["m"], s["q"], s["u"])
        return w if kind == "winding" else (w, gx, gn, gm, gq)
    if kind == "treepm":
        a, gx, gm = _gravity(s["x"], s["m"], s["w"], c["softening"] ** 2, c["r_split"], float(c["cells"]),
                             "full" if c["adjoint"] else "none")
        return (a, gx, gm) if c["adjoint"] else a
    eps2 = c["softening"] ** 2
    if kind in ("octree8_step", "direct_step"):
        a, gx, gm = _gravity(s["x"], s["m"], s["w"], eps2 + 1e-12, 0.0 if c["cutoff"] > 1e5 else c["cutoff"],
                             1.0 if c.get("periodic") else 0.0, "query")
        return a, gx, gm
    if kind == "forest_adjoint":
        parts, at = [], 0
        for k in s["sizes"]:
            parts.append(_gravity(s["x"][at:at + k], s["m"][at:at + k], s["w"][at:at + k], eps2))
            at += k
        return tuple(torch.cat([p[i] for p in parts]) for i in range(3))
    if kind == "gravity_force":
        return _gravity(s["x"], s["m"], None, eps2, adjoint="none")[0]
    a, gx, gm = _gravity(s["x"], s["m"], s["w"], eps2)
    if kind == "stochastic_step":
        return a, None, None  # the gradients hold the draws fixed
    return a, gx, gm
