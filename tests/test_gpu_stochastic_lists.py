"""The native stochastic estimator where its lists run over: more draws than one
refinement takes (128), and coarse cuts with more weighted nodes than the list
holds (2,048), which are listed range by range."""
import numpy as np
import pytest

import sbh_b200 as B
import sbh_oracle as O
import sbh_workloads as W
from conftest import rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,beta,coarse,samples", [(3000, 2.0, 1.0, 128), (3000, 2.0, 1.0, 129),
                                                   (3000, 2.0, 0.75, 1024),
                                                   (60000, 9.0, 4.0, 32), (60000, 9.0, 4.0, 200)])
def test_draws_and_cuts_past_the_lists_match_oracle(cuda, n, beta, coarse, samples):
    """Same draws as the oracle's restatement; tolerances as at the usual sizes
    (rows 3e-5, gradients 1e-4). At beta 9 over 4 a group's cut holds some 4,000
    weighted nodes at 60,000 particles."""
    p, m = W.plummer(n, seed=n)
    t = B.NativeTree().build(p, m, leaf_size=16)
    _, perm, rec = t.export()
    sp = np.ascontiguousarray(np.concatenate([p[perm], m[perm, None]], axis=1), np.float32)
    kw = dict(beta=beta, beta_coarse=coarse, samples=samples, seed=21, softening=1e-2)
    got = t.stochastic_force(**kw).cpu().numpy()
    want, _, walks = O.native_stochastic(sp, perm, rec, group_size=B.native_group_size(), expectation=False, **kw)
    assert walks > 0
    assert rel_l2(got, want) < 3e-5
    if n > 10000:
        return
    w = np.random.default_rng(1).normal(size=p.shape).astype(np.float32)
    _, gx, gm = t.stochastic_force_vjp(w, want_force=False, **kw)
    T = O.NativeTree(p, m, leaf_size=16)
    assert T.stochastic_plan(rec, group_size=B.native_group_size(), **kw) > 0
    dx, dm = T.adjoint(w, 1e-2, quad=True)
    assert rel_l2(gx.cpu().numpy(), dx) < 1e-4
    assert rel_l2(gm.cpu().numpy(), dm) < 1e-4
