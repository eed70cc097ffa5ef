"""Forests of more than 512 systems, whose small ones are walked by one warp per
group (up to 64 particles while the forest has few groups, up to 1,536 where it has
many), against the same systems walked by several warps."""
import numpy as np
import pytest
import torch

import sbh_b200 as B
import sbh_workloads as W
from conftest import rel_l2

pytestmark = pytest.mark.gpu

SIZES = [64, 65, 1, 100, 0, 129, 700, 1536, 1537, 33, 2500, 2]


def _rows(p, m, w, sizes, **kw):
    off = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int64)
    t = B.NativeTree().build(p[:off[-1]], m[:off[-1]], None, off, leaf_size=8, group_size=kw.pop("group", 128))
    mono = dict(beta=2.0, softening=1e-2, cutoff=0.5, quadrupole=False)
    st = dict(beta=2.0, beta_coarse=1.0, softening=1e-2, samples=kw.pop("samples", 32), seed=5)
    w = w[:off[-1]]
    out = [t.force(beta=2.0, softening=1e-2), *t.force_vjp(w, beta=2.0, softening=1e-2), t.force(**mono),
           *t.force_vjp(w, **mono), t.stochastic_force(**st), *t.stochastic_force_vjp(w, **st)]
    return [v.cpu().numpy() for v in out], t


@pytest.mark.parametrize("others", [600, 4000])
@pytest.mark.parametrize("group,samples", [(128, 32), (64, 200), (96, 33)])
def test_one_warp_per_group_matches_several(cuda, others, group, samples):
    """The same systems alone and in front of a forest of many: the same
    plans and draws (their particles keep their indices), FP32 sums of up to
    2,500 terms in another order. Every system has to agree, empty ones among them."""
    n = sum(SIZES)
    tail = [5] * others  # 4,000: more than 24 groups per SM
    p, m = W.plummer(n + sum(tail), seed=3)
    rng = np.random.default_rng(4)
    m = (m * rng.uniform(0.5, 1.5, len(m))).astype(np.float32)
    w = rng.normal(size=p.shape).astype(np.float32)
    few, _ = _rows(p, m, w, SIZES, group=group, samples=samples)
    many, _ = _rows(p, m, w, SIZES + tail, group=group, samples=samples)
    off = np.concatenate([[0], np.cumsum(SIZES)])
    for a, b in zip(few, many):
        assert np.isfinite(b).all()
        for s, e in zip(off[:-1], off[1:]):
            if e - s > 1:
                assert rel_l2(b[s:e], a[s:e]) < 5e-6, (s, e)


def test_small_systems_match_pairwise_sums(cuda):
    """3,000 systems of 20 particles, every pair opened: force and gradients against
    FP64 pair sums (20 terms in FP32: 1e-6 and 2e-6)."""
    k, n = 3000, 20
    rng = np.random.default_rng(7)
    p = rng.random((k, n, 3)).astype(np.float32)
    m = (rng.random((k, n)) + 0.5).astype(np.float32)
    w = rng.normal(size=(k, n, 3)).astype(np.float32)
    t = B.NativeTree().build(p.reshape(-1, 3), m.reshape(-1), None, np.arange(k + 1, dtype=np.int64) * n, leaf_size=4)
    f, gx, gm = (v.cpu().numpy() for v in t.force_vjp(w.reshape(-1, 3), beta=1e4, softening=1e-2))
    r = (p[:, :, None] - p[:, None]).astype(np.float64)
    ir = ((r * r).sum(-1) + 1e-4 + 1e-12) ** -0.5
    ir[:, np.arange(n), np.arange(n)] = 0.0
    W2, M = w.astype(np.float64), m.astype(np.float64)[:, None]
    rw = (r * W2[:, :, None]).sum(-1)
    q = M[..., None] * ((3.0 * ir ** 5 * rw)[..., None] * r - (ir ** 3)[..., None] * W2[:, :, None])
    want = -(M[..., None] * (ir ** 3)[..., None] * r).sum(2), q.sum(2) - q.sum(1), -(ir ** 3 * rw).sum(1)
    for got, ref, tol in zip((f, gx, gm), want, (1e-6, 2e-6, 2e-6)):
        assert rel_l2(got.reshape(ref.shape), ref) < tol
    assert t.stats()["groups"] == k


def test_forest_walks_in_a_graph(cuda):
    """Both launches of a forest's walk captured and replayed on new cotangents."""
    sizes = SIZES + [7] * 600
    off = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int64)
    p, m = W.plummer(int(off[-1]), seed=9)
    w = [torch.tensor(np.random.default_rng(k).normal(size=p.shape).astype(np.float32), device=cuda) for k in (1, 2)]
    t = B.NativeTree().build(p, m, None, off, leaf_size=8)
    held = w[0].clone()
    want = [[v.clone() for v in t.force_vjp(x, beta=2.0)] for x in w]
    s = torch.cuda.Stream()
    with torch.cuda.stream(s):
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=s):
            out = t.force_vjp(held, beta=2.0)
    for k in (0, 1, 0):
        held.copy_(w[k])
        torch.cuda.synchronize()
        g.replay()
        torch.cuda.synchronize()
        for a, b in zip(out, want[k]):  # the node-side sums meet in atomics, in any order
            assert rel_l2(a.cpu().numpy(), b.cpu().numpy()) < 2e-6
