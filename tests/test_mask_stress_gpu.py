"""Masked calls back to back, without a pause between them: every result has the bits of the first, waited-for one."""
import pytest
import torch

import fused_attention_b200 as fa
from fused_attention_b200 import _lib

pytestmark = pytest.mark.gpu

ONE, PAIR = _lib.FLAG_FORCE_PIPELINED | _lib.FLAG_NO_PAIR, _lib.FLAG_FORCE_PAIR


@pytest.mark.parametrize("H,B,R,L,flags", [(128, 2, 40, 3072, 0), (128, 1, 40, 4095, 0), (128, 2, 20, 1920, ONE), (128, 2, 40, 2048, PAIR),
                                           (64, 8, 16, 2048, 0), (64, 8, 16, 1024, 0), (64, 2, 30, 1999, 0), (32, 8, 16, 1024, 0)])
def test_mask_buffers_are_not_refilled_under_a_reader(H, B, R, L, flags):
    """A mask tile's buffer is handed back before the exponentials, and the next tile or half tile is on its way at once:
    a thread whose reads were not complete by then would take the next tile's values."""
    g = torch.Generator(device="cuda")
    g.manual_seed(L + H)
    q, k, v = (torch.randn(B, L, R * H, generator=g, device="cuda").half() for _ in range(3))
    mask = torch.triu(torch.full((L, L), float("-inf"), device="cuda", dtype=torch.float16), diagonal=1)
    mask = mask.unsqueeze(0).repeat(B, 1, 1)
    first = fa.attention_forward(H, 32, q, k, v, mask, flags=flags | _lib.FLAG_SYNC)
    for _ in range(6):
        outs = [fa.attention_forward(H, 32, q, k, v, mask, flags=flags) for _ in range(6)]
        torch.cuda.synchronize()
        assert all(torch.equal(first, y) for y in outs)
    assert fa.read_status(0) == (0, 0)


@pytest.mark.parametrize("H,R,flags", [(16, 40, 0), (32, 40, 0), (64, 30, 0), (128, 20, _lib.FLAG_NO_PAIR)])
def test_calls_behind_a_launch_that_found_no_work(H, R, flags):
    """A planned call with an aligned mask ends with a launch that leaves at once: small calls right behind it, whose CTAs
    take its place on the SMs, have the bits they have alone."""
    g = torch.Generator(device="cuda")
    g.manual_seed(H)
    B, L = 2, 2048
    q, k, v = (torch.randn(B, L, R * H, generator=g, device="cuda").half() for _ in range(3))
    small = [torch.randn(64, 48, 4 * 32, generator=g, device="cuda").half() for _ in range(3)]
    tile = [torch.randn(16, 300, 4 * 64, generator=g, device="cuda").half() for _ in range(3)]
    mask = torch.triu(torch.full((L, L), float("-inf"), device="cuda", dtype=torch.float16), diagonal=1)
    mask = mask.unsqueeze(0).repeat(B, 1, 1)
    calls = (lambda: fa.attention_forward(H, 32, q, k, v, mask, flags=flags), lambda: fa.attention_forward(32, 32, *small),
             lambda: fa.attention_forward(64, 32, *tile))
    first = []
    for call in calls:
        first.append(call())
        torch.cuda.synchronize()
    for _ in range(20):
        outs = [call() for call in calls]
        torch.cuda.synchronize()
        assert all(torch.equal(a, b) for a, b in zip(first, outs))
    assert fa.read_status(0) == (0, 0)
