"""Work items cut into exactly three parts: the schedule (CPU) and the results (GPU)."""
import pytest
import torch

import fused_attention_b200 as fa
from fused_attention_b200 import _lib

ONE = _lib.FLAG_FORCE_PIPELINED | _lib.FLAG_NO_PAIR
# key steps that are and are not a multiple of three, the fewest and the most items, a full round before the divided one
SHAPES = [(1, 4, 3000, 128), (1, 1, 8192, 128), (1, 3, 4096, 128), (1, 4, 1500, 128), (1, 2, 2048, 64), (1, 1, 1600, 64),
          (1, 1, 8192, 64), (1, 20, 2048, 64), (1, 3, 1700, 64)]


@pytest.mark.parametrize("B,R,L,H", SHAPES)
def test_every_item_has_exactly_three_parts(B, R, L, H):
    sched = fa.describe_schedule(B, L, R * H, H, flags=ONE)
    n, n_items = sched["key_steps"], -(-L // 256) * R * B
    assert sched["tail_grid"] == 3 * sched["tail_items"] > 0
    seen = {}
    for cta in range(sched["grid"]):
        for item, j0, ln in fa.cta_segments(sched, n_items, cta):
            for j in range(j0, j0 + ln):
                assert (item, j) not in seen
                seen[(item, j)] = cta
    assert len(seen) == n_items * n
    for item in range(sched["full_rounds"] * sched["grid"], n_items):
        parts = sorted({seen[(item, j)] for j in range(n)})
        assert len(parts) == 3 and parts == list(range(parts[0], parts[0] + 3))


@pytest.mark.gpu
@pytest.mark.parametrize("B,R,L,H", SHAPES + [(1, 4, 2048, 32), (1, 2, 2000, 16)])
def test_thirds_give_the_undivided_result(B, R, L, H):
    """Bounds as in test_parity_gpu.py: 2e-3 and 2e-4 against fp32 attention, a quarter of it against whole items."""
    g = torch.Generator(device="cuda")
    g.manual_seed(L + R)
    q, k, v = (torch.randn(B, L, R * H, generator=g, device="cuda").half() for _ in range(3))
    mask = torch.zeros(B, L, L, device="cuda", dtype=torch.float16)
    mask[:, :, L // 2:] = float("-inf")
    mask[:, ::7, :] = 0
    qf, kf, vf = (t.float().view(B, L, R, H).transpose(1, 2) for t in (q, k, v))
    for m in (None, mask):
        call = lambda flags=0: fa.attention_forward(H, 32, q, k, v, m, flags=flags | _lib.FLAG_SYNC)
        y = call()
        assert torch.equal(y, call()) and torch.isfinite(y).all()
        s = qf @ kf.mT / H ** 0.5
        ref = (torch.softmax(s if m is None else s + m.float()[:, None], -1) @ vf).transpose(1, 2).reshape(B, L, R * H)
        d = (y.float() - ref).abs()
        assert float(d.max()) <= 2e-3 and float(d.mean()) <= 2e-4, (float(d.max()), float(d.mean()))
        assert float((y.float() - call(_lib.FLAG_NO_SPLIT).float()).abs().max()) <= 5e-4
    assert fa.read_status(0) == (0, 0)
