"""Planned calls, aligned masks: which items look through the K and V of key tiles that other items leave out.

Results: the bits of the call without a plan.  Which kernel had the call follows from the mask alone: a key tile with a value
that is not finite, which some items leave out and others work on, gives the call to the kernel behind the planned one."""
import pytest
import torch

import fused_attention_b200 as fa
from fused_attention_b200 import _lib
from fused_attention_b200.workloads import make_inputs
from test_mask_gpu import _recorded, status_word_stays_clear  # noqa: F401

pytestmark = pytest.mark.gpu

TILE, PAIR = 128, 256


def mask_of(kind, B, L):
    rows, keys = torch.arange(L)[:, None], torch.arange(L)[None, :]
    if kind == "blocks":   # every other key tile of every other pair of query tiles, shifted by one from entry to entry
        gone = [((rows // PAIR) + (keys // TILE) + b) % 2 == 1 for b in range(B)]
    else:
        gone = [{"causal": keys > rows, "reversed causal": keys < rows, "band": (keys - rows).abs() > 300}[kind]] * B
    return torch.where(torch.stack(gone), float("-inf"), 0.0).half()


@pytest.mark.parametrize("value", [float("inf"), float("nan")])
@pytest.mark.parametrize("where", ["k", "v"])
@pytest.mark.parametrize("tile", ["first", "middle", "last"])
@pytest.mark.parametrize("kind", ["causal", "reversed causal", "band", "blocks"])
@pytest.mark.parametrize("H,R,L", [(32, 28, 2176), (64, 30, 2056), (128, 30, 2048), (16, 30, 2048)])
def test_every_key_tile_that_some_items_leave_out_is_looked_through(H, R, L, kind, tile, where, value):
    """Neighbours before and behind, the last pair with one query tile (2176 keys are 17 tiles) or with a ragged one (2056),
    the first and the last column of a head, the first and the last row of a key tile."""
    B = 2
    n = (L + TILE - 1) // TILE
    route = fa.describe_call(B, L, R * H, H, 16)
    assert route["planned"] and route["launches"] == 3 and fa.stream_has_scratch()
    q, k, v = (t.cuda() for t in make_inputs(B, L, R * H, 1.0, L))
    mask = mask_of(kind, B, L)
    kt = {"first": 0, "middle": n // 2, "last": n - 1}[tile]
    row, column = (kt * TILE, 7 * H) if where == "k" else (min(kt * TILE + TILE, L) - 1, 8 * H - 1)
    {"k": k, "v": v}[where][1, row, column] = value
    pairs = torch.nn.functional.pad(mask[1, :, kt * TILE:kt * TILE + TILE], (0, 0, 0, -L % PAIR), value=float("-inf"))
    left_out = (pairs == float("-inf")).reshape(-1, PAIR * pairs.shape[1]).all(1)
    mask = mask.cuda()
    y = fa.attention_forward(H, 32, q, k, v, mask, flags=_lib.FLAG_SYNC)
    assert fa.plan_taken() is not bool(left_out.any() and not left_out.all())
    plain = _recorded(q, k, v, H, mask, _lib.FLAG_NO_SPLIT)
    assert bool((~torch.isfinite(plain)).any())
    assert torch.equal(torch.nan_to_num(y, nan=9.0), torch.nan_to_num(plain, nan=9.0))
