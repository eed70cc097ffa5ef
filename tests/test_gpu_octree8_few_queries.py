"""octree8 traversals of few queries in trees too large for shared units (more
than 16,384 particles): a warp takes one query up to 2,368 of them, four up to
4,095, then 32."""
import numpy as np
import pytest
import torch

import sbh_b200 as B

pytestmark = pytest.mark.gpu


def _call(cuda, n, nq, depth):
    """call(vjp, ordered, prune, periodic) -> rows, for uniform particles and queries."""
    rng = np.random.default_rng(n + nq)
    p, q = rng.random((n, 3), dtype=np.float32), torch.tensor(rng.random((nq, 3), dtype=np.float32), device=cuda)
    w = torch.tensor(rng.normal(size=(nq, 3)).astype(np.float32), device=cuda)
    leaf, node = B.build_octree8_buffers(p, np.zeros_like(p), np.full(n, 1.0 / n, np.float32),
                                         np.zeros(3, np.float32), np.ones(3, np.float32), max_depth=depth)
    L, s = B.lib(), torch.cuda.current_stream(cuda).cuda_stream
    ws = {True: torch.empty(int(L.sbh_traversal_ordered_workspace_bytes(nq)), dtype=torch.uint8, device=cuda),
          False: torch.empty(int(L.sbh_traversal_workspace_bytes()), dtype=torch.uint8, device=cuda)}
    args = (leaf.data_ptr(), leaf.numel(), node.data_ptr(), node.numel(), q.data_ptr(), nq)

    def call(vjp, ordered, prune=0, periodic=0):
        out = torch.full((nq, 3), float("nan"), device=cuda)
        tail = (out.data_ptr(), 2.0, 1e-2, 0.4 if prune else 1e7, prune, 2.0, periodic, 1.0, 256,
                ws[ordered].data_ptr(), ws[ordered].numel())
        if vjp:
            assert L.sbh_barnes_hut_force_octree8_soft_vjp(s, *args, w.data_ptr(), *tail) == 0
        else:
            assert L.sbh_barnes_hut_force_octree8_soft(s, *args, *tail) == 0
        return out

    call.keep = (leaf, node, q, w)  # `args` holds addresses only
    call.status = lambda: max(B.read_device_status(v) for v in ws.values())
    return call


@pytest.mark.parametrize("nq", [64, 2368, 2369, 2371, 4095, 4096])
def test_rows_do_not_depend_on_queries_per_warp(cuda, nq):
    """Bit for bit those of one thread per query."""
    call = _call(cuda, 20000, nq, 5)
    for vjp in (False, True):
        for prune, periodic in ((0, 0), (1, 0), (1, 1)):
            a, b = call(vjp, True, prune, periodic), call(vjp, False, prune, periodic)
            assert torch.equal(a, b) and not torch.isnan(a).any()
    assert call.status() == 0


def test_few_queries_far_apart_are_no_slower_in_order(cuda):
    """64 queries over 200,000 particles: with 32 of them on one stack the sorted
    order took 4 times as long as one thread per query; now it takes a third."""
    call = _call(cuda, 200000, 64, 6)
    ms = {}
    for ordered in (True, False):
        call(False, ordered)
        for _ in range(3):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            call(False, ordered)
            b.record()
            b.synchronize()
            ms[ordered] = min(a.elapsed_time(b), ms.get(ordered, 1e9))
    assert ms[True] < ms[False], ms
