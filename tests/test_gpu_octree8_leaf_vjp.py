"""Unsoftened stochastic VJP where every subdomain is a leaf (depth 3 or less), so
that the estimate is the plain sum over leaves, at the counts around the four
particles loaded at a time."""
import numpy as np
import pytest
import torch

import sbh_b200 as B
from conftest import rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,depth", [(1, 1), (3, 1), (4, 1), (5, 1), (40, 1), (2100, 3), (9001, 3), (700, 2)])
@pytest.mark.parametrize("periodic", [False, True])
def test_leaf_sums_of_the_gravity_vjp(cuda, n, depth, periodic):
    """Against the FP64 gradient of sum -m r / (|r| + 0.1)^3; sums of at most 9,001
    terms, one running FP32 sum: 5e-6."""
    rng = np.random.default_rng(n)
    p, q = rng.random((n, 3), dtype=np.float32), rng.random((300, 3), dtype=np.float32)
    m, w = (rng.random(n) + 0.5).astype(np.float32) / n, rng.normal(size=(300, 3)).astype(np.float32)
    leaf, node = B.build_octree8_buffers(p, np.zeros_like(p), m, np.zeros(3, np.float32), np.ones(3, np.float32),
                                         max_depth=depth)
    kw = dict(beta=1.0, samples_per_subdomain=1, seed=2, periodic=periodic, box_length=1.0)
    got = B.stochastic_barnes_hut_force_octree8_vjp(leaf, node, q, w, **kw).cpu().numpy()
    Q = torch.tensor(q, dtype=torch.float64, requires_grad=True)
    r = Q[:, None] - torch.tensor(p, dtype=torch.float64)[None]
    if periodic:
        r = r - torch.floor(r.detach() + 0.5)
    d = (r * r).sum(-1).sqrt()
    f = -(torch.tensor(m, dtype=torch.float64)[None, :, None] * r / ((d + 0.1) ** 3)[..., None]).sum(1)
    want, = torch.autograd.grad(f, Q, torch.tensor(w, dtype=torch.float64))
    assert rel_l2(got, want.numpy()) < 5e-6
