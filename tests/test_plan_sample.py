"""Which tiles of a mask are looked at to find out whether planning the call pays, without a GPU."""
import ctypes

import numpy as np
import pytest

from fused_attention_b200 import _lib

MAX_GROUPS, MOST = 1024, 256   # pairs of query tiles of all batch entries that are planned for, tiles that are looked at


def samples(B, n):
    lib, out = _lib.load(), (ctypes.c_uint32 * 4)()
    assert lib.fa_b200_describe_plan_sample(B, 128 * n, 0, out) == _lib.OK
    rows = []
    for i in range(out[3]):
        assert lib.fa_b200_describe_plan_sample(B, 128 * n, i, out) == _lib.OK
        rows.append(tuple(out))
    assert lib.fa_b200_describe_plan_sample(B, 128 * n, len(rows), out) == _lib.ERR_SHAPE
    b, q, k, count = np.array(rows, dtype=np.int64).T
    assert (count == len(rows)).all() and b.max() < B and q.max() < n and k.max() < n
    return b, q, k


def masks(B, n):
    """Which tiles begin with -inf: a function of batch entry, query tile and key tile."""
    spread = n * (0.25 + 0.75 * np.arange(1, B + 1) / B)
    shuffled = np.random.default_rng(B * n).permutation(spread)
    return {
        "causal": lambda b, q, k: k > q,
        "reversed causal": lambda b, q, k: k < q,
        "padding": lambda b, q, k: (k >= spread[b]) | (q < 0),
        "padding, shuffled": lambda b, q, k: (k >= shuffled[b]) | (q < 0),
        "band": lambda b, q, k: abs(k - q) * 4 > n,
        "causal window": lambda b, q, k: (k > q) | ((q - k) * 4 > n),
    }


@pytest.mark.parametrize("first", range(16, 257, 40))
def test_the_sample_judges_a_mask_as_all_of_its_tiles_do(first):
    """For every number of key tiles and of batch entries that can be planned, the share of -inf among the tiles that are
    looked at is that of all tiles.  (The largest difference over these masks and others is 0.053; the rule's line lies at
    a fifth, and the masks that a plan is for are well above it.)"""
    for n in range(first, min(first + 40, 257)):
        for B in range(1, MAX_GROUPS // ((n + 1) // 2) + 1):
            at = samples(B, n)
            every = np.ix_(np.arange(B), np.arange(n), np.arange(n))
            for name, neg in masks(B, n).items():
                share, of_all = neg(*at).mean(), np.broadcast_to(neg(*every), (B, n, n)).mean()
                assert abs(share - of_all) <= 0.1, (name, B, n, share, of_all)


def test_few_tiles_are_all_looked_at():
    for B, n in ((1, 16), (1, 2), (3, 5), (4, 8), (256, 1)):
        assert sorted(zip(*(x.tolist() for x in samples(B, n)))) == [(b, q, k) for b in range(B) for q in range(n) for k in range(n)]
    assert len(samples(2, 16)[0]) == MOST


def test_sizes_without_a_plan_are_refused():
    out = (ctypes.c_uint32 * 4)()
    for B, L in ((0, 128), (1, 0), (1, 257 * 128), (1025, 128), (1, 2 ** 32 - 1)):
        assert _lib.load().fa_b200_describe_plan_sample(B, L, 0, out) == _lib.ERR_SHAPE
    assert _lib.load().fa_b200_describe_plan_sample(1, 128, 0, None) == _lib.ERR_NULL_POINTER
