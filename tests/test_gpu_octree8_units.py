"""The octree8 traversals whose sums are taken in units (trees of at most 16,384
particles) and the single-block sort, at the edges of their ranges."""
import numpy as np
import pytest
import torch

import sbh_b200 as B
import sbh_oracle as O
import sbh_workloads as W
from conftest import rel_l2

pytestmark = pytest.mark.gpu


# 16,384 particles are the last in units; fewer than 64 queries stay unordered
@pytest.mark.parametrize("n,nq,depth", [(1, 64, 1), (7, 100, 2), (600, 63, 3), (600, 64, 3), (2000, 1001, 5),
                                        (16384, 300, 6), (16385, 300, 6)])
def test_rows_do_not_depend_on_how_warps_share_the_tree(cuda, n, nq, depth):
    """The ordered workspace (warps sharing the units of 32 queries) against the
    small one (one thread per query), bit for bit; force and VJP against the oracle's
    FP64 sums of the same decisions (FP32 sums of at most 16,385 terms: 1e-5), so a
    unit left out or counted twice shows; the force against the direct sum within
    the opening error."""
    rng = np.random.default_rng(n)
    p = rng.random((n, 3), dtype=np.float32)
    m = (rng.random(n) + 0.5).astype(np.float32) / n
    lo, hi = np.zeros(3, np.float32), np.ones(3, np.float32)
    leaf, node = B.build_octree8_buffers(p, np.zeros_like(p), m, lo, hi, max_depth=depth)
    q = rng.random((nq, 3), dtype=np.float32)
    w = rng.normal(size=q.shape).astype(np.float32)
    Q, C = torch.tensor(q, device=cuda), torch.tensor(w, device=cuda)
    L = B.lib()
    s = torch.cuda.current_stream(cuda).cuda_stream
    big = torch.empty(int(L.sbh_traversal_ordered_workspace_bytes(nq)), dtype=torch.uint8, device=cuda)
    small = torch.empty(int(L.sbh_traversal_workspace_bytes()), dtype=torch.uint8, device=cuda)
    args = (leaf.data_ptr(), leaf.numel(), node.data_ptr(), node.numel(), Q.data_ptr(), nq)
    for cutoff, prune, per in ((0.4, 1, 0), (1e7, 0, 0), (0.4, 1, 1)):
        tail = (2.0, 1e-2, cutoff, prune, 2.0, per, 1.0, 256)
        rows = []
        for ws in (big, small):
            f, g = (torch.full((nq, 3), float("nan"), device=cuda) for _ in range(2))
            assert L.sbh_barnes_hut_force_octree8_soft(s, *args, f.data_ptr(), *tail, ws.data_ptr(), ws.numel()) == 0
            assert L.sbh_barnes_hut_force_octree8_soft_vjp(s, *args, C.data_ptr(), g.data_ptr(), *tail, ws.data_ptr(),
                                                           ws.numel()) == 0
            assert B.read_device_status(ws) == 0
            rows.append((f, g))
        assert torch.equal(rows[0][0], rows[1][0]) and torch.equal(rows[0][1], rows[1][1])
        okw = dict(eps=1e-2, cutoff=cutoff, prune_enabled=bool(prune), prune_r_cut_mult=2.0, periodic=bool(per))
        for got, kernel, cot in zip(rows[0], (O.KERNEL_SOFT, O.KERNEL_SOFT_VJP), (None, w)):
            want, _ = O.bh_octree8(leaf.cpu().numpy(), node.cpu().numpy(), q, 2.0, kernel, cot=cot, **okw)
            assert rel_l2(got.cpu().numpy(), want) < 1e-5
        if not prune:
            want = O.direct_force_soft(p, m, q, 1e-2, cutoff, False, 1.0)
            assert rel_l2(rows[0][0].cpu().numpy(), want) < (5e-6 if n < 16 else 2e-2)


@pytest.mark.parametrize("n", [1, 31, 32, 33, 1023, 1024, 1025, 5000, 16383, 16384, 16385])
def test_sorts_around_the_single_block_limit(cuda, n):
    """Keys in order, equal keys in input order, the permutation complete."""
    p, m = W.uniform_cube(n, seed=n)
    p[n // 2:] = p[: n - n // 2]  # every position twice or so
    t = B.NativeTree().build(p, m, leaf_size=16)
    keys, perm, _ = t.export()
    assert np.array_equal(np.sort(perm), np.arange(n, dtype=perm.dtype))
    assert (keys[1:] >= keys[:-1]).all()
    same = keys[1:] == keys[:-1]
    assert (perm[1:][same] > perm[:-1][same]).all()
    arr = O.NativeTree(p, m, leaf_size=16).arrays()
    np.testing.assert_array_equal(keys, arr["keys"])
    np.testing.assert_array_equal(perm.astype(np.int64), arr["perm"])


@pytest.mark.parametrize("copies", [2, 8, 9, 40])
def test_small_sorts_with_keys_that_agree_in_their_top_bits(cuda, copies):
    """Clusters far below the resolution of a key's top 32 bits (about 2^-11 of
    the box per axis): runs up to the limit of the in-place pass and past it."""
    rng = np.random.default_rng(copies)
    centres = rng.random((3000 // copies, 3))
    p = (np.repeat(centres, copies, axis=0) + rng.uniform(-2e-6, 2e-6, (3000 // copies * copies, 3)))
    p = p.astype(np.float32)[rng.permutation(3000 // copies * copies)]
    m = np.full(len(p), 1.0 / len(p), np.float32)
    keys, perm, _ = B.NativeTree().build(p, m, leaf_size=8).export()
    arr = O.NativeTree(p, m, leaf_size=8).arrays()
    np.testing.assert_array_equal(keys, arr["keys"])
    np.testing.assert_array_equal(perm.astype(np.int64), arr["perm"])
