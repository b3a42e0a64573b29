"""Sequences of at most 160 keys, most of them on the kernel of small CTAs, against the CPU oracle.

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


def check(y, expected):
    assert torch.equal(torch.isnan(y), torch.isnan(expected))
    m = error_metrics(torch.nan_to_num(y), torch.nan_to_num(expected))
    assert m["max_abs"] <= MAX_ABS_TOL and m["mean_abs"] <= MEAN_ABS_TOL, m


# tiles of 16 rows, two at a time: either side of each multiple of 16 and 32
@pytest.mark.parametrize("L", [1, 2, 15, 16, 17, 31, 32, 33, 48, 49, 63, 64, 65, 81, 96, 97, 100, 113, 127, 128, 129, 144, 145, 160])
@pytest.mark.parametrize("H", [16, 32, 64, 128])
def test_short_sequences(H, L):
    q, k, v = make_inputs(3, L, 5 * H, 1.0, H + L)
    dev = [t.cuda() for t in (q, k, v)]
    y = fa.attention_forward(H, 32, *dev, flags=_lib.FLAG_SYNC)
    check(y.float().cpu(), oracle(q, k, v, H))
    host = fa.attention_forward_host(H, 32, q, k, v)
    assert torch.equal(y.cpu(), host)
    # masks at every start within 16 bytes, at the very beginning and end of their allocation, rows without a key
    gen = torch.Generator().manual_seed(L)
    mask = torch.randn(3, L, L, generator=gen).half()
    mask[0] += torch.triu(torch.full((L, L), float("-inf")), diagonal=1).half()
    mask[1, L // 2] = float("-inf")
    mask[2, :, : L // 2] = float("-inf")
    want = oracle(q, k, v, H, mask)
    for offset in (0, 1, 2, 3, 4, 8):
        store = torch.full((offset + mask.numel(),), float("nan"), dtype=torch.float16, device="cuda")
        on_gpu = store[offset:].view_as(mask)
        on_gpu.copy_(mask)
        check(fa.attention_forward(H, 32, *dev, on_gpu, flags=_lib.FLAG_SYNC).float().cpu(), want)


def test_large_scores_and_values_that_are_not_finite():
    B, R, L, H = 2, 3, 50, 64
    q, k, v = make_inputs(B, L, R * H, 1.0, 3)
    check(fa.attention_forward(H, 32, (40 * q).cuda(), (40 * k).cuda(), v.cuda(), flags=_lib.FLAG_SYNC).float().cpu(),
          oracle(40 * q, 40 * k, v, H))
    for where in range(3):
        for value in (float("inf"), float("nan")):
            x = [t.clone() for t in (q, k, v)]
            x[where][1, 7, H + 5] = value
            dev = [t.cuda() for t in x]
            y = fa.attention_forward(H, 32, *dev, flags=_lib.FLAG_SYNC)
            one = fa.attention_forward(H, 32, *dev, flags=_lib.FLAG_SYNC | _lib.FLAG_FORCE_SIMPLE)
            assert torch.equal(torch.isnan(y), torch.isnan(one)) and torch.equal(torch.isinf(y), torch.isinf(one))
