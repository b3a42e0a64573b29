"""Host buffers cut into blocks of query rows: the bits of one device call with whole work items."""
import os
import subprocess
import sys

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


FOUR_STREAMS = """
import torch, fused_attention_b200 as fa
from fused_attention_b200 import _lib
from fused_attention_b200.workloads import make_inputs
B, R, L, H = 8, 2, 1021, 64
fa.attention_forward_host(H, 32, *make_inputs(B, L, R * H, 1.0, 1), torch.triu(torch.full((L, L), float("-inf")), 1).half().repeat(B, 1, 1))
q, k, v = (t.cuda() for t in make_inputs(1, 3000, 4 * 128, 1.0, 2))
torch.cuda.synchronize()
outs, streams = [], [torch.cuda.Stream() for _ in range(4)]
for s in streams:
    with torch.cuda.stream(s):
        outs.append(fa.attention_forward(128, 32, q, k, v))
torch.cuda.synchronize()
whole = fa.attention_forward(128, 32, q, k, v, flags=_lib.FLAG_NO_SPLIT | _lib.FLAG_SYNC)
assert not torch.equal(outs[0], whole)
assert all(torch.equal(outs[0], y) for y in outs[1:])
"""


def test_host_calls_leave_the_scratch_to_the_callers_streams():
    """Four streams of a device get scratch for divided and planned calls; masked host calls take none of it (in a process
    of its own, where no stream has any yet)."""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    subprocess.run([sys.executable, "-c", FOUR_STREAMS], check=True, cwd=root, timeout=300)
