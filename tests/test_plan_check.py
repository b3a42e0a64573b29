"""Which pair of query tiles looks through the K and V of a key tile that other pairs leave out, without a GPU."""
import ctypes

import numpy as np
import pytest

from fused_attention_b200 import _lib

NONE = 0xFFFF


def checker(works, kt):
    out = (ctypes.c_uint32 * 1)()
    assert _lib.load().fa_b200_describe_plan_check(len(works), works.astype(np.uint8).tobytes(), kt, out) == _lib.OK
    return out[0]


def pairs_that_keep(works):
    return np.pad(works, ((0, len(works) % 2), (0, 0))).reshape(-1, 2, works.shape[1]).any(1)


def patterns(n):
    """works[query tile, key tile] of several masks."""
    q, k = np.arange(n)[:, None], np.arange(n)[None, :]
    rng = np.random.default_rng(n)
    yield from (k <= q, k >= q, abs(k - q) <= 2, (q // 2 + k) % 2 == 0, k + 0 * q < n // 2, k + 0 * q < 0, k + 0 * q >= 0)
    yield from (rng.random((n, n)) < share for share in (0.05, 0.3, 0.9))


@pytest.mark.parametrize("n", [1, 2, 3, 16, 17, 31, 256])
def test_one_pair_that_works_on_a_key_tile_looks_it_through(n):
    for works in patterns(n):
        keeps, who = pairs_that_keep(works), np.array([checker(works[:, kt], kt) for kt in range(n)])
        mixed = keeps.any(0) & ~keeps.all(0)
        assert ((who != NONE) == mixed).all()
        assert keeps[who[mixed], np.nonzero(mixed)[0]].all()


@pytest.mark.parametrize("n", [16, 32, 64])
def test_no_pair_has_most_of_the_looking_to_do(n):
    """Random blocks of 256 x 128, half of them left out: about two key tiles a pair."""
    works = np.repeat(np.random.default_rng(1).random((n // 2, n)) < 0.5, 2, axis=0)
    who = [checker(works[:, kt], kt) for kt in range(n)]
    assert max(np.bincount([w for w in who if w != NONE])) <= 10


def test_refused():
    out, call = (ctypes.c_uint32 * 1)(), _lib.load().fa_b200_describe_plan_check
    assert call(2, None, 0, out) == call(2, b"\1\1", 0, None) == _lib.ERR_NULL_POINTER
    assert call(0, b"", 0, out) == call(257, bytes(257), 0, out) == call(2, b"\1\1", 2, out) == _lib.ERR_SHAPE
