"""The cooperative tree walks at the edges of their shapes: group sizes around
the slot boundaries, both numbers of warps per group, leaves longer than a
batch (coincident points), source counts around a batch, and single queries."""
import numpy as np
import pytest

import sbh_b200 as B
import sbh_oracle as O
import sbh_workloads as W
from conftest import rel_l2

pytestmark = pytest.mark.gpu


def _system(n, seed):
    """n particles, the last fifth of them copies of one point when n >= 200."""
    p, m = W.plummer(n, seed=seed)
    rng = np.random.default_rng(seed)
    if n >= 200:
        p[-n // 5:] = p[0]
    m = (m * rng.uniform(0.5, 1.5, n)).astype(np.float32)
    return p, m, rng.normal(size=p.shape).astype(np.float32)


# group 8 puts 11,000 particles above the rule's 12 groups per SM (4 warps per
# group), the others below it (16 warps per group)
@pytest.mark.parametrize("n,group", [(1, 128), (2, 128), (31, 128), (33, 64), (129, 128), (300, 32), (1000, 33),
                                     (1000, 65), (2500, 97), (2500, 128), (11000, 8)])
@pytest.mark.parametrize("short_range", [False, True])
def test_walks_match_oracle_at_edges(cuda, n, group, short_range):
    """Force and full adjoint against the oracle's FP64 evaluation of the same
    plan. Tolerances as for the larger systems (FP32 sums of at most 11,000
    terms: 1e-5 for the force, 1e-4 for the gradients)."""
    p, m, w = _system(n, 100 + n)
    kw = dict(beta=2.0, softening=1e-2)
    if short_range:
        kw.update(cutoff=0.5, quadrupole=False)
    t = B.NativeTree().build(p, m, leaf_size=8, group_size=group)
    f_alone = t.force(**kw).cpu().numpy()
    f, gx, gm = (v.cpu().numpy() for v in t.force_vjp(w, **kw))
    T = O.NativeTree(p, m, leaf_size=8)
    with O.native_quadrupole_linear(0.0 if short_range else 0.5):
        T.plan(2.0, group)
    ekw = dict(cutoff=0.5) if short_range else dict(quad=True)
    want, _ = T.force(1e-2, **ekw)
    dx, dm = T.adjoint(w, 1e-2, **ekw)
    if n == 1:
        assert not f.any() and not f_alone.any() and not want.any()
        return
    assert rel_l2(f_alone, want) < 1e-5
    assert rel_l2(f, want) < 1e-5
    assert rel_l2(gx, dx) < 1e-4
    assert rel_l2(gm, dm) < 1e-4


@pytest.mark.parametrize("n,nq", [(1, 1), (2, 31), (31, 33), (33, 65), (300, 129), (5000, 1000)])
def test_winding_walks_match_oracle_at_edges(cuda, n, nq):
    """Winding number and its adjoint; half of the queries outside the tree's
    box, one of them on a source (d = 0)."""
    p, nrm, m = W.ellipsoid_surface(n, seed=n)
    rng = np.random.default_rng(nq)
    q = rng.uniform(-2.0, 2.0, (nq, 3)).astype(np.float32)
    q[0] = p[0]
    u = rng.normal(size=nq).astype(np.float32)
    t = B.NativeTree().build(p, m, normals=nrm, leaf_size=8)
    w_alone = t.winding_number(q).cpu().numpy()
    w, gq, gp, gn, gm = (v.cpu().numpy() for v in t.winding_number_vjp(q, u, want_value=True))
    T = O.NativeTree(p, m, leaf_size=8)
    T.wn_plan(q, 2.0)
    want = T.wn_eval(nrm)
    dq, dp, dn, dm = T.wn_adjoint(nrm, u)
    scale = max(np.linalg.norm(want), 1e-6)
    assert np.linalg.norm(w_alone - want) < 1e-5 * scale and np.linalg.norm(w - want) < 1e-5 * scale
    for got, ref in ((gq, dq), (gp, dp), (gn, dn), (gm, dm)):
        assert np.linalg.norm(got - ref) < 1e-4 * max(np.linalg.norm(ref), 1e-6)
