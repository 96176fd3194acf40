"""Trees, openings and FRI tails at the edges of their kernels' shapes.

The reduce launch hashes a level of 128 nodes by threads and smaller ones by
quads of lanes, in stages of 8 levels over blocks of 256; deeper trees start
with leaf subtrees and node kernels down to 2^16 hashes.  Openings take eight
lanes per (query, stored-level group), four pairs per warp.  The line folds of
at most 2048 values share one launch: a cluster of eight blocks down to 512
values, one block from 256."""
import numpy as np
import pytest

import test_tree_plan as tree_plan
from gpu_util import to_dev
from vortexstark_b200 import prover, tune
from vortexstark_b200.merkle import FusedRoot, MerkleTree
from vortexstark_b200.workload import m31_array

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ncols", [1, 4, 5])
@pytest.mark.parametrize("log_n", list(range(1, 20)) + [21])
def test_roots_at_every_depth(oracle, log_n, ncols):
    cols = [m31_array(31 * log_n + i, 1 << log_n) for i in range(ncols)]
    want = tuple(oracle.merkle_root(cols).tolist())
    d = [to_dev(c) for c in cols]
    for k in (1, 2, 3, 4) if log_n > 16 else (0,):
        tune.set_leaf_k(log_n, k)
        try:
            assert FusedRoot(log_n).commit(d) == want, k
        finally:
            tune.set_leaf_k(log_n, 0)


@pytest.mark.parametrize("ncols", [1, 4, 7])
@pytest.mark.parametrize("log_n", [1, 5, 9, 10, 11, 14, 20, 21])
def test_root_only_through_the_launchers(oracle, log_n, ncols):
    cols = [m31_array(17 * log_n + i, 1 << log_n) for i in range(ncols)]
    assert MerkleTree.commit_root_only([to_dev(c) for c in cols], log_n) == tuple(oracle.merkle_root(cols).tolist())


def test_the_plan_is_the_one_that_is_built():
    """vx_tree_plan describes this device's trees, with its own rule and with a
    subtree size that was set, and every such plan holds."""
    from vortexstark_b200 import _lib
    for depth in range(1, 32):
        for k in (0, 1, 2, 3, 4):
            tune.set_leaf_k(depth, k)
            try:
                heights, top, n_cnt, words = tree_plan.plan(depth)
                assert words == _lib.lib().vx_merkle_workspace_words(depth)
                if depth > 16:
                    assert heights[1] == tune.get(tune.LEAF_K, depth)[0] == (k or min(max(depth - 18, 1), 4))
                if k == 0:
                    tree_plan.test_tree_plan_shape(depth)
                tree_plan.check_levels(depth)
                if 16 <= depth <= 22:
                    tree_plan.simulate_reduce(depth, heights, top, n_cnt, k)
            finally:
                tune.set_leaf_k(depth, 0)


def _least_words(depth, k=4):
    """Words of the plan that stores least: 2^k-leaf subtrees, 16 -> 1 node
    levels while more than 2^20 hashes are left, every 4th height above."""
    heights = [k]
    while depth - heights[-1] > 20:
        heights.append(heights[-1] + 4)
    left = max(depth - heights[-1] - 8, 0)
    while heights[-1] < depth:
        heights.append(min(heights[-1] + 4, depth))
    counters = 0
    while left > 0:
        step = min(left, 8)
        counters += 1 << (left - step)
        left -= step
    return sum(8 << (depth - h) for h in heights) + counters


@pytest.mark.parametrize("log_n", [17, 18, 20, 21, 22, 23, 24, 25, 26])
def test_root_in_a_small_workspace(oracle, log_n):
    """A workspace of the least words of that plan is enough (some depths take less)."""
    import ctypes as C

    import torch

    from vortexstark_b200 import _lib
    col = m31_array(7 + log_n, 1 << log_n)
    want = tuple(oracle.merkle_root([col]).tolist())
    d = to_dev(col)
    ptrs = (C.c_void_p * 1)(d.data_ptr())
    words = _least_words(log_n)
    work = torch.empty(words, dtype=torch.int32, device="cuda")
    root = torch.empty(8, dtype=torch.int32, device="cuda")
    call = _lib.lib().vx_merkle_root_cols
    assert call(ptrs, 1, log_n, work.data_ptr(), words, root.data_ptr(), None) == 0
    assert tuple(int(x) for x in root.cpu().numpy().view(np.uint32)) == want
    assert call(ptrs, 1, log_n, work.data_ptr(), words // 2, root.data_ptr(), None) == 1
    _lib.clear_error()


@pytest.mark.parametrize("log_n,blowup,nq", [(4, 1, 1), (4, 1, 3), (4, 3, 17), (5, 2, 4), (6, 3, 5), (7, 2, 33),
                                             (8, 1, 2), (9, 1, 31), (10, 2, 79), (11, 3, 1), (13, 1, 7), (15, 3, 81)])
def test_proofs_at_odd_query_counts(oracle, log_n, blowup, nq):
    a, b = 1000 + log_n, 77 * nq
    assert prover.prove_bytes(a, b, log_n, blowup, nq) == oracle.prove(a, b, log_n, blowup, nq)


@pytest.mark.parametrize("log_n,first", [(8, 8), (9, 9), (10, 10), (11, 11), (14, 11)])
def test_fri_tails_while_the_device_is_full(oracle, log_n, first):
    """Tails that start at 2^first values (above 2^8: on a cluster), several at
    once beside larger proofs, so that a cluster's blocks start when others
    leave room for them."""
    import torch
    assert first == min(log_n, 11)
    jobs = [(log_n, 40 + i, 3 * i) for i in range(6)] + [(18, 7, 9), (18, 8, 10)]
    work = [(prover.ProverCache(k), torch.cuda.Stream(), k, a, b) for k, a, b in jobs]
    want = [oracle.prove(a, b, k) for k, a, b in jobs]
    for _ in range(4):
        for cache, stream, _, a, b in reversed(work):
            cache.prove_async(a, b, stream.cuda_stream)
        torch.cuda.synchronize()
        assert [w[0].result_bytes() for w in work] == want
    for w in work:
        w[0].close()
