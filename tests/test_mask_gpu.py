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


def _recorded(q, k, v, H, mask, flags):
    """The same call recorded into a CUDA graph and replayed: a stream that is being captured gets no plan."""
    fa.attention_forward(H, 32, q, k, v, mask, flags=flags)          # set-up outside the capture
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        y = fa.attention_forward(H, 32, q, k, v, mask, flags=flags)
    graph.replay()
    torch.cuda.synchronize()
    return y


def _block_mask(B, L, kind):
    """Masks whose 128 x 128 tiles are of every kind: -inf throughout, zero throughout, neither."""
    gen = torch.Generator().manual_seed(B * L)
    rows, keys = torch.arange(L)[:, None], torch.arange(L)[None, :]
    m = torch.zeros(B, L, L)
    if kind == "causal":
        m[:, (keys > rows)] = float("-inf")
    elif kind == "padding":
        for b in range(B):
            m[b, :, max(1, L * (b + 1) // (B + 1)):] = float("-inf")
    elif kind == "left_padding":
        for b in range(B):
            m[b, :, :L * (b + 1) // (B + 2)] = float("-inf")
    elif kind == "band":
        m[:, ((keys - rows).abs() > 100)] = float("-inf")
    elif kind == "dense":
        m = 0.5 * torch.randn(B, L, L, generator=gen)
    else:
        for b in range(B):                     # every tile of a kind of its own; whole pairs of query tiles without a key
            for i in range(0, L, 128):
                for j in range(0, L, 128):
                    pick = int(torch.randint(0, 4, (1,), generator=gen))
                    tile = m[b, i:i + 128, j:j + 128]
                    if pick == 0 or (b == 0 and i < 256):
                        tile.fill_(float("-inf"))
                    elif pick == 1:
                        tile.copy_(torch.randn(tile.shape, generator=gen))
                    elif pick == 2:
                        tile[::3] = float("-inf")
    return m.half()


@pytest.mark.parametrize("B,R,L,H", [(4, 40, 301, 32), (3, 50, 265, 16), (5, 80, 201, 64), (2, 32, 1021, 64), (2, 20, 1101, 128),
                                     (1, 2, 515, 64), (2, 30, 1928, 64), (2, 30, 2048, 32), (3, 20, 1944, 128), (2, 30, 2048, 128)])
@pytest.mark.parametrize("kind", ["causal", "padding", "left_padding", "band", "dense", "tiles"])
def test_planned_masks(B, R, L, H, kind):
    """Calls that are planned: key tiles that the mask takes away are left out, tiles that are zero or -inf are not
    fetched, rows on no 16-byte boundary are copied.  The same bits as without a plan, and the oracle's values."""
    route = fa.describe_call(B, L, R * H, H, 16)
    assert route["planned"] == (L != 201) and fa.stream_has_scratch()      # (two key tiles are not worth a plan)
    assert route["launches"] == (1 if L == 201 else 3 if L % 8 == 0 else 2)
    q, k, v = make_inputs(B, L, R * H, 1.0, L)
    mask = _block_mask(B, L, kind)
    dev = [t.cuda() for t in (q, k, v, mask)]
    y = fa.attention_forward(H, 32, *dev, flags=_lib.FLAG_SYNC)
    assert torch.equal(torch.nan_to_num(y, nan=9.0), torch.nan_to_num(_recorded(*dev[:3], H, dev[3], _lib.FLAG_NO_SPLIT), nan=9.0))
    cols = slice((R - 1) * H, R * H)
    assert_close(y[..., cols].float().cpu(), oracle(*(t[..., cols].contiguous() for t in (q, k, v)), H, mask))


@pytest.mark.parametrize("B,R,L,H", [(16, 4, 2048, 64), (32, 2, 1928, 32), (8, 2, 4096, 128), (4, 1, 8192, 64), (12, 6, 2048, 64)])
@pytest.mark.parametrize("kind", ["causal", "padding"])
def test_large_batches_keep_their_plan(B, R, L, H, kind):
    """Numbers of batch entries and of key tiles whose product is a multiple of 256, and one whose is not: what is looked at to
    find out whether a mask leaves enough out has to come from all of its key tiles."""
    assert fa.describe_call(B, L, R * H, H, 16)["planned"] and fa.stream_has_scratch()
    q, k, v = (t.cuda() for t in make_inputs(B, L, R * H, 1.0, L))
    mask = _block_mask(B, L, kind).cuda()
    y = fa.attention_forward(H, 32, q, k, v, mask, flags=_lib.FLAG_SYNC)
    assert fa.plan_taken() is True
    assert torch.equal(y, _recorded(q, k, v, H, mask, _lib.FLAG_NO_SPLIT))


@pytest.mark.parametrize("value", [float("inf"), float("nan")])
@pytest.mark.parametrize("where", ["k", "v", "q"])
@pytest.mark.parametrize("B,R,L", [(2, 30, 2048), (3, 40, 515)])
def test_masked_keys_that_are_not_finite_are_not_left_out(where, value, B, R, L):
    """0 * inf and inf - inf are NaN: a masked key with an infinity or a NaN in K or V reaches the result with a plan
    exactly as it does without one."""
    H = 64
    assert fa.describe_call(B, L, R * H, H, 16)["planned"] and fa.stream_has_scratch()
    q, k, v = (t.cuda() for t in make_inputs(B, L, R * H, 1.0, L))
    mask = torch.zeros(B, L, L, dtype=torch.float16)
    mask[:, :, 200:] = float("-inf")
    mask = mask.cuda()
    {"q": q, "k": k, "v": v}[where][1, 450, 7 * H + 3] = value
    y = fa.attention_forward(H, 32, q, k, v, mask, flags=_lib.FLAG_SYNC)
    plain = _recorded(q, k, v, H, mask, _lib.FLAG_NO_SPLIT)
    assert torch.equal(torch.isnan(y), torch.isnan(plain)) and bool(torch.isnan(y).any())
    assert torch.equal(torch.nan_to_num(y, nan=9.0), torch.nan_to_num(plain, nan=9.0))


@pytest.mark.parametrize("value", [float("inf"), float("-inf"), float("nan")])
@pytest.mark.parametrize("where", ["k", "v"])
@pytest.mark.parametrize("H,R,L", [(32, 30, 2048), (64, 30, 2048), (128, 30, 1928), (64, 40, 515)])
def test_keys_that_only_some_items_leave_out_and_that_are_not_finite(where, value, H, R, L):
    """Causal: the key tile is worked on by some items and left out by others.  Where its rows start on 16-byte boundaries
    the items that work on it find the value, and the kernel behind the planned one does the call again."""
    B = 2
    assert fa.describe_call(B, L, R * H, H, 16)["planned"] and fa.stream_has_scratch()
    q, k, v = (t.cuda() for t in make_inputs(B, L, R * H, 1.0, L))
    mask = torch.full((L, L), float("-inf"), dtype=torch.float16).triu(1).repeat(B, 1, 1).cuda()
    {"k": k, "v": v}[where][1, L - 70, 7 * H + 3] = value
    y = fa.attention_forward(H, 32, q, k, v, mask, flags=_lib.FLAG_SYNC)
    plain = _recorded(q, k, v, H, mask, _lib.FLAG_NO_SPLIT)
    assert torch.equal(torch.nan_to_num(y, nan=9.0), torch.nan_to_num(plain, nan=9.0))
    assert bool((~torch.isfinite(plain)).any())


@pytest.mark.parametrize("B,R,L,H", [(2, 30, 2048, 64), (2, 30, 1928, 128), (3, 40, 1021, 64), (2, 30, 2048, 32), (2, 9, 389, 128)])
def test_rows_that_are_runs_of_zeros(B, R, L, H):
    """Rows of a tile as runs: ends on and beside the edges of words, halves and tiles, rows without a key, -0 in a run; and
    one row that is no run, which makes its tile a mask tile.  The bits of the call without a plan."""
    assert fa.describe_call(B, L, R * H, H, 16)["planned"] and fa.stream_has_scratch()
    q, k, v = (t.cuda() for t in make_inputs(B, L, R * H, 1.0, L))
    ends = torch.tensor([0, 1, 2, 31, 32, 33, 63, 64, 65, 95, 96, 97, 126, 127, 128, 129, 200, 256, L - 1, L])
    gen = torch.Generator().manual_seed(L + H)
    a, b = (ends[torch.randint(0, len(ends), (B, L, 1), generator=gen)] for _ in range(2))
    keys = torch.arange(L)
    mask = torch.where((keys >= torch.minimum(a, b)) & (keys < torch.maximum(a, b)), 0.0, float("-inf")).half()
    mask[:, ::7] = torch.where(mask[:, ::7] == 0, torch.tensor(-0.0, dtype=torch.float16), mask[:, ::7])
    mask[0, 300, :] = 0.0
    mask[0, 300, 40:50] = float("-inf")
    mask = mask.cuda()
    y = fa.attention_forward(H, 32, q, k, v, mask, flags=_lib.FLAG_SYNC)
    plain = _recorded(q, k, v, H, mask, _lib.FLAG_NO_SPLIT)
    assert torch.equal(torch.nan_to_num(y, nan=9.0), torch.nan_to_num(plain, nan=9.0))
