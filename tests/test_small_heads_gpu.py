"""Head dimensions 16 and 32 on the warp-specialised kernel, against the CPU oracle.

Tolerance as in test_parity_gpu.py: max-abs <= 2e-3 and mean-abs <= 2e-4 against the fp32 oracle on the same
fp16-rounded inputs.
"""
import pytest
import torch

import fused_attention_b200 as fa
from fused_attention_b200 import _lib
from fused_attention_b200.workloads import make_inputs
from oracle.naive_attention import MAX_ABS_TOL, MEAN_ABS_TOL, attention as oracle, error_metrics

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def status_word_stays_clear():
    yield
    assert fa.read_status(0) == (0, 0)


# one key step more than the one-tile kernel's share, tile edges, many items per CTA, last rounds divided in two and three
@pytest.mark.parametrize("B,R,L", [(1, 1, 257), (2, 3, 383), (1, 3, 384), (2, 2, 385), (1, 5, 1000), (40, 16, 130), (20, 10, 300),
                                   (1, 4, 2048), (1, 3, 2600), (3, 31, 2049)])
@pytest.mark.parametrize("H", [16, 32])
def test_warp_specialised_kernel_at_small_head_dims(B, R, L, H):
    q, k, v = make_inputs(B, L, R * H, 1.0, L + H)
    dev = [t.cuda() for t in (q, k, v)]
    y = fa.attention_forward(H, 16, *dev, flags=_lib.FLAG_SYNC)
    assert torch.equal(y, fa.attention_forward(H, 16, *dev, flags=_lib.FLAG_SYNC))
    whole = fa.attention_forward(H, 16, *dev, flags=_lib.FLAG_SYNC | _lib.FLAG_NO_SPLIT)
    one_tile = fa.attention_forward(H, 16, *dev, flags=_lib.FLAG_SYNC | _lib.FLAG_FORCE_SIMPLE)
    bh = [(b, h) for b in (0, B - 1) for h in (0, R - 1)]     # the oracle on the corners, the one-tile kernel on the rest
    for b, h in bh:
        cols = slice(h * H, (h + 1) * H)
        want = oracle(q[b:b + 1, :, cols].contiguous(), k[b:b + 1, :, cols].contiguous(), v[b:b + 1, :, cols].contiguous(), H)
        for got in (y, whole):
            m = error_metrics(got[b:b + 1, :, cols].float().cpu(), want)
            assert m["max_abs"] <= MAX_ABS_TOL and m["mean_abs"] <= MEAN_ABS_TOL, m
    for got in (y, whole):   # (two results within MAX_ABS_TOL of the same value)
        assert float((got.float() - one_tile.float()).abs().max()) <= 2 * MAX_ABS_TOL
