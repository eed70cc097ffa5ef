"""Scans at the tile counts where one block stops carrying the total: two tiles
of 512 moment vectors, eight of 2,048 words."""
import numpy as np
import pytest

import sbh_b200 as B
import sbh_oracle as O
import sbh_workloads as W
from conftest import rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [511, 512, 1023, 1024, 1025, 4096, 4097, 16385])
def test_moment_and_adjoint_scans_at_tile_edges(cuda, n):
    """Node moments (build) and the gradients pushed down from the nodes (one more
    element than particles) against the oracle's FP64 sums of the same plan."""
    p, m = W.plummer(n, seed=n)
    w = np.random.default_rng(n).normal(size=p.shape).astype(np.float32)
    f, gx, gm = (v.cpu().numpy() for v in B.NativeTree().build(p, m, leaf_size=8).force_vjp(w, beta=2.0,
                                                                                            softening=1e-2))
    T = O.NativeTree(p, m, leaf_size=8)
    with O.native_quadrupole_linear(0.5):
        T.plan(2.0, 128)
    want, _ = T.force(1e-2, quad=True)
    dx, dm = T.adjoint(w, 1e-2, quad=True)
    assert rel_l2(f, want) < 1e-5
    assert rel_l2(gx, dx) < 1e-4
    assert rel_l2(gm, dm) < 1e-4
