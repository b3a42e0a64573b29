"""Unaligned planned masks on both sides of the line between passing rows on as runs of zeros and as mask tiles."""
import pytest
import torch

import fused_attention_b200 as fa
from fused_attention_b200 import _lib
from fused_attention_b200.workloads import make_inputs
from test_mask_gpu import _block_mask, _recorded, status_word_stays_clear  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["causal", "padding", "band", "tiles"])
@pytest.mark.parametrize("H,B,R,L", [(64, 2, 49, 515), (64, 2, 50, 515), (32, 7, 21, 385), (32, 4, 37, 387), (16, 8, 12, 387), (128, 2, 9, 389)])
def test_bits_of_the_call_without_a_plan(H, B, R, L, kind):
    """B R pairs of query tiles: 294 and 300, 294 and 296 (two items per SM), 192; head_dim 128 whatever their number."""
    assert fa.describe_call(B, L, R * H, H, 2)["planned"] and fa.stream_has_scratch()
    q, k, v = (t.cuda() for t in make_inputs(B, L, R * H, 1.0, L))
    mask = _block_mask(B, L, kind).cuda()
    y = fa.attention_forward(H, 32, q, k, v, mask, flags=_lib.FLAG_SYNC)
    assert fa.plan_taken() is True
    assert torch.equal(torch.nan_to_num(y, nan=9.0), torch.nan_to_num(_recorded(q, k, v, H, mask, _lib.FLAG_NO_SPLIT), nan=9.0))
