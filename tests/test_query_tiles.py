"""The order in which prompt attention gets its tiles of queries (ft_attn_prefill_order_tiles): a permutation of the caller's list, the tiles that take
longest at its end where the tcgen05 kernel runs, the caller's own order where the mma.sync kernel does."""
import random

import numpy as np
import pytest

from fasttalk_llm_microservice_b200 import native as N


def ordered(lens, pos0, nq, nkv, d, rows=None):
    starts = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    pos = np.array(pos0, np.int32)
    tiles = [(r, q0) for r, n in enumerate(lens) for q0 in range(0, n, 64)]
    req, q0 = (np.array([t[i] for t in tiles], np.int32) for i in (0, 1))
    rc = N.load().ft_attn_prefill_order_tiles(starts.ctypes.data, pos.ctypes.data, req.ctypes.data, q0.ctypes.data, len(tiles), nq, nkv, d,
                                              int(starts[-1]) if rows is None else rows)
    tc = (nq // nkv in (3, 4)) and d in (64, 128) and (rows is None or rows > 0)
    assert rc == int(tc and any(min(64, lens[r] - q) <= 32 and (pos0[r] + min(lens[r], q + 64) - 1) // 64 + 1 >= 4 for r, q in tiles))
    return tiles, list(zip(req.tolist(), q0.tolist()))


def key_tiles(lens, pos0, t):
    r, q0 = t
    rows = min(64, lens[r] - q0)
    n = (pos0[r] + q0 + rows - 1) // 64 + 1
    return n / 2 if rows <= 32 and n >= 4 else n


MIXED = ([2048, 300, 64, 900, 17, 600], [0, 2000, 5000, 0, 4000, 100])


@pytest.mark.parametrize("nq,nkv,d,rows", [(8, 8, 64, None), (16, 2, 64, None), (16, 8, 128, None), (32, 8, 64, 0), (32, 8, 128, -1), (32, 8, 96, None)])
def test_the_mma_sync_kernel_gets_the_callers_order(nq, nkv, d, rows):
    for lens, pos0 in (MIXED, ([500] * 12, [0] * 12), ([30] * 64, [100] * 64)):
        given, got = ordered(lens, pos0, nq, nkv, d, rows)
        assert got == given


@pytest.mark.parametrize("nq,nkv,d", [(32, 8, 64), (24, 8, 128), (32, 8, 128), (4, 1, 64)])
def test_long_tiles_stand_last_and_nothing_is_lost(nq, nkv, d):
    rng = random.Random(nq + d)
    cases = [MIXED, ([211] * 6, [5000] * 6), ([1], [0]), ([2048] * 4, [0] * 4), ([64] * 70, [0] * 70)]
    cases += [([rng.randint(1, 900) for _ in range(n)], [rng.choice([0, 5, 63, 64, 700, 9000]) for _ in range(n)]) for n in (1, 2, 7, 33)]
    for lens, pos0 in cases:
        given, got = ordered(lens, pos0, nq, nkv, d)
        assert sorted(got) == sorted(given)
        work = [key_tiles(lens, pos0, t) for t in got]
        # later tiles are shorter by no more than what is sorted by: an eighth of an SM's share, or four key tiles (and the halves' own start)
        slack = max(4, sum(w + 6 for w in work) * nkv / 148 / 8) + 1
        longest = 0
        for w in work:
            assert w > longest - slack
            longest = max(longest, w)
    given, got = ordered(*MIXED, nq, nkv, d)
    assert got[-1] == (2, 0)                   # 64 queries behind 5000 keys


def test_tiles_that_differ_little_keep_their_requests_together():
    given, got = ordered([100] * 40, [600] * 40, 32, 8, 128)
    assert got == given


def test_no_tiles_and_missing_lists():
    lib = N.load()
    assert lib.ft_attn_prefill_order_tiles(0, 0, 0, 0, 0, 32, 8, 64, 10) == 0
    assert lib.ft_attn_prefill_order_tiles(0, 0, 0, 0, 3, 32, 8, 64, 10) != 0
