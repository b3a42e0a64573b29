"""Host buffers cut into blocks of query rows: the bits of one device call with whole work items."""
import pytest
import torch

import fused_attention_b200 as fa
from fused_attention_b200 import _lib
from fused_attention_b200.workloads import make_inputs

pytestmark = pytest.mark.gpu


# a last block of one row, of fewer rows than a tile, one row short of a block; two blocks and eight; every mask path
@pytest.mark.parametrize("B,R,L,H", [(1, 24, 1025, 128), (2, 32, 600, 64), (1, 32, 2047, 64), (3, 40, 1300, 32), (1, 16, 2048, 128),
                                     (1, 40, 513, 64), (4, 48, 511, 128)])
@pytest.mark.parametrize("masked", [False, True])
def test_blocks_of_query_rows(B, R, L, H, masked):
    q, k, v = make_inputs(B, L, R * H, 1.0, L + H)
    mask = None
    if masked:
        mask = torch.triu(torch.full((L, L), float("-inf")), diagonal=1).half().unsqueeze(0).repeat(B, 1, 1)
        mask[:, :, : L // 3] += torch.randn(B, L, L // 3, generator=torch.Generator().manual_seed(L)).half()
    want = fa.attention_forward(H, 32, q.cuda(), k.cuda(), v.cuda(), None if mask is None else mask.cuda(), flags=_lib.FLAG_NO_SPLIT)
    assert torch.equal(want.cpu(), fa.attention_forward_host(H, 32, q, k, v, mask))
    assert fa.read_status(0) == (0, 0)
