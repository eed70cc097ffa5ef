"""The direct sums' splits at their edges: warps, tiles of 512 sources, chunks
of 32, and the query counts where the split changes."""
import numpy as np
import pytest
import torch

import sbh_b200 as B
import sbh_oracle as O
from conftest import rel_l2

pytestmark = pytest.mark.gpu


# 37,888 and 151,552 queries fill a wave of blocks with 4 warps and one per query set
@pytest.mark.parametrize("n,nq", [(1, 1), (31, 33), (33, 31), (511, 512), (513, 65), (1025, 1000), (517, 37888),
                                  (517, 37889), (70, 151552), (70, 151553)])
@pytest.mark.parametrize("cutoff,periodic", [(1e7, False), (0.3, False), (60.0, False), (0.3, True), (1e7, True)])
def test_direct_sums_match_float64_at_edges(cuda, n, nq, cutoff, periodic):
    """cutoff 1e7: no pair attenuated; 60: the att = 1 radius (0.23) cuts through
    the box, so both forms run; 0.3: nearly every pair attenuated. FP32 sums of
    at most 1,025 terms: 2e-6."""
    rng = np.random.default_rng(n + nq)
    p = rng.random((n, 3), dtype=np.float32)
    m = (rng.random(n) + 0.5).astype(np.float32) / n
    q = rng.random((nq, 3), dtype=np.float32)
    q[0] = p[0]
    w = rng.normal(size=(nq, 3)).astype(np.float32)
    kw = dict(softening_scale=1e-2, cutoff_scale=cutoff, periodic=periodic, box_length=1.0)
    f = B.softened_direct_force(p, m, q, **kw).cpu().numpy()
    g = B.softened_direct_force_vjp(p, m, q, w, **kw).cpu().numpy()
    want = O.direct_force_soft(p, m, q, 1e-2, cutoff, periodic, 1.0)
    want_g = O.direct_force_soft_vjp(p, m, q, w, 1e-2, cutoff, periodic, 1.0)
    scale = max(np.linalg.norm(want), 1e-30)
    assert np.linalg.norm(f - want) < 2e-6 * scale + 1e-7 * (n == 1)
    assert rel_l2(g, want_g) < 2e-6


# 9,472 queries are the last that take 16 warps whatever the sources; 290 and 130 leave
# 4 warps chunks of unequal number, 40 one, 4,100 sources keep 16 at 37,889 queries
@pytest.mark.parametrize("n,nq", [(1025, 9472), (290, 9473), (130, 30000), (40, 37000), (4100, 37889)])
@pytest.mark.parametrize("cutoff,periodic", [(60.0, False), (0.3, True)])
def test_direct_splits_match_float64(cuda, n, nq, cutoff, periodic):
    """As above, sums of at most 4,100 terms."""
    test_direct_sums_match_float64_at_edges(cuda, n, nq, cutoff, periodic)


def test_direct_sums_without_sources(cuda):
    q = torch.rand(40, 3, device=cuda)
    e = torch.empty(0, 3, device=cuda)
    assert not B.softened_direct_force(e, e[:, 0], q).any()
