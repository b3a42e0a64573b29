"""Additive masks on the warp-specialised kernels: how their tiles come in, against the CPU oracle.

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

ONE = _lib.FLAG_FORCE_PIPELINED | _lib.FLAG_NO_PAIR


@pytest.fixture(autouse=True)
def status_word_stays_clear():
    yield
    assert fa.read_status(0) == (0, 0)


def run(q, k, v, H, mask, flags=0):
    return fa.attention_forward(H, 32, q.cuda(), k.cuda(), v.cuda(), mask, flags=flags | _lib.FLAG_SYNC).float().cpu()


def assert_close(y, expected):
    assert torch.equal(torch.isnan(y), torch.isnan(expected))
    m = error_metrics(torch.nan_to_num(y), torch.nan_to_num(expected))
    assert m["max_abs"] <= MAX_ABS_TOL and m["mean_abs"] <= MEAN_ABS_TOL, m


@pytest.mark.parametrize("H", [16, 32, 64, 128])
@pytest.mark.parametrize("L", [1, 2, 127, 129, 131, 255, 257, 388, 390, 391, 1021])
@pytest.mark.parametrize("offset", [0, 1, 2, 3, 4])
def test_mask_rows_that_tma_cannot_fetch(H, L, offset):
    """Every start of a row within its 8 bytes, the mask at the very beginning and the very end of its allocation,
    rows whose last word reaches behind the mask."""
    q, k, v = make_inputs(2, L, 3 * H, 1.0, 50 + L)
    gen = torch.Generator().manual_seed(L)
    mask = (0.5 * torch.randn(2, L, L, generator=gen)).half()
    mask[0] += torch.triu(torch.full((L, L), float("-inf")), diagonal=1).half()
    store = torch.full((offset + mask.numel(),), float("nan"), dtype=torch.float16, device="cuda")
    on_gpu = store[offset:].view_as(mask)
    on_gpu.copy_(mask)
    assert_close(run(q, k, v, H, on_gpu, ONE if H >= 64 else 0), oracle(q, k, v, H, mask))


@pytest.mark.parametrize("H,flags", [(32, 0), (64, ONE), (128, ONE), (128, _lib.FLAG_FORCE_PAIR)])
def test_rows_whose_first_tiles_are_masked_and_whose_scores_are_far_below_zero(H, flags):
    """Left padding of more than a key tile, and scores around -40 in the exp2 domain: against a reference of 0 instead
    of the row's own maximum every P would be lost in fp16."""
    B, L = 2, 520
    q, k, v = make_inputs(B, L, 2 * H, 1.0, 7)
    q = q.abs() * 0 + 1.0
    k = k * 0.25 - 28.0 / H ** 0.5                     # q.k / sqrt(H) around -28
    mask = torch.zeros(B, L, L, dtype=torch.float16)
    mask[0, :, :130] = float("-inf")
    mask[1, :, :400] = float("-inf")
    assert_close(run(q, k, v, H, mask.cuda(), flags), oracle(q, k, v, H, mask))
