"""The tensor-core Hamming shortlist: lists equal to the CPU restatement's where ranges,
tiles and blocks end, with crowded distances, and where the candidates overflow."""
import numpy as np
import pytest

import oracle as O
import psift

pytestmark = pytest.mark.gpu


def _check(q, c, k, ctx=None):
    gi, gd = psift.hamming_topk(q, c, k, ctx=ctx)
    ri, rd = O.hamming_topk(q, c, k)
    np.testing.assert_array_equal(gd, rd)
    np.testing.assert_array_equal(gi, ri)


# the first 2048 codes are listed directly; then 512-code blocks, 256-code tiles, 128-query
# tiles, ranges of 8x
@pytest.mark.parametrize("nq,ncat,k", [(1, 1, 1), (3, 40, 64), (5, 2047, 64), (5, 2048, 64), (1, 2049, 64),
                                       (127, 2305, 7), (128, 2561, 64), (129, 16384, 33), (65, 16385, 1),
                                       (300, 131073, 64), (64, 262657, 64), (1000, 300000, 16)])
def test_lists_equal_the_oracle(nq, ncat, k):
    rng = np.random.default_rng(nq + ncat)
    c = rng.integers(0, 2 ** 64, (ncat, 2), dtype=np.uint64)
    q = rng.integers(0, 2 ** 64, (nq, 2), dtype=np.uint64)
    q[: nq // 2] = c[rng.integers(0, ncat, nq // 2)] ^ np.uint64(5)  # near duplicates
    _check(q, c, k)


def test_query_blocks():
    # 8192 queries are taken at a time
    rng = np.random.default_rng(2)
    c = rng.integers(0, 2 ** 64, (3000, 2), dtype=np.uint64)
    _check(rng.integers(0, 2 ** 64, (8200, 2), dtype=np.uint64), c, 5)


def test_crowded_distances():
    # few distinct codes: most distances tie, the index decides
    rng = np.random.default_rng(3)
    pool = rng.integers(0, 2 ** 64, (7, 2), dtype=np.uint64)
    c = pool[rng.integers(0, 7, 70001)]
    q = np.concatenate([pool[rng.integers(0, 7, 60)], rng.integers(0, 2 ** 64, (40, 2), dtype=np.uint64)])
    _check(q, c, 64)
    _check(q, np.zeros_like(c), 64)
    _check(np.zeros_like(q), ~np.zeros_like(c), 64)


def test_candidates_that_overflow():
    # every code of the last third is nearer to the first queries than all before it
    rng = np.random.default_rng(4)
    c = rng.integers(0, 2 ** 64, (90000, 2), dtype=np.uint64)
    q = rng.integers(0, 2 ** 64, (80, 2), dtype=np.uint64)
    noise = np.uint64(1) << rng.integers(0, 64, 30000, dtype=np.uint64)
    c[60000:, 0] = q[0, 0] ^ noise
    c[60000:, 1] = q[0, 1]
    q[1] = q[0]
    q[2] = ~q[0]
    ctx = psift.Context(0)
    for k in (1, 40, 64):
        _check(q, c, k, ctx)
    ctx.close()


def test_query_blocks_of_a_full_device():
    # 8192 queries need 68 MB of scratch; with 32 MB left they are taken 1024 at a time
    import ctypes as C

    import torch
    rng = np.random.default_rng(5)
    c = rng.integers(0, 2 ** 64, (5000, 2), dtype=np.uint64)
    q = rng.integers(0, 2 ** 64, (8192, 2), dtype=np.uint64)
    _check(q[:4], c, 8)  # the kernels are loaded
    ctx = psift.Context(0)
    dq, dc = (torch.from_numpy(a.view(np.int64)).cuda() for a in (q, c))
    idx, dist = (torch.zeros((len(q), 8), dtype=torch.int32, device="cuda") for _ in range(2))
    free = torch.cuda.mem_get_info()[0]
    fill = torch.empty(free - (32 << 20), dtype=torch.uint8, device="cuda")
    try:
        ctx.check(ctx.lib.psift_hamming_topk_dev(ctx.handle, C.c_void_p(dq.data_ptr()), len(q),
                                                 C.c_void_p(dc.data_ptr()), len(c), 8, C.c_void_p(idx.data_ptr()),
                                                 C.c_void_p(dist.data_ptr())))
        ctx.synchronize()
    finally:
        del fill
        torch.cuda.empty_cache()
    ri, rd = O.hamming_topk(q, c, 8)
    np.testing.assert_array_equal(idx.cpu().numpy().view(np.uint32), ri)
    np.testing.assert_array_equal(dist.cpu().numpy().view(np.uint32), rd)
    ctx.close()
