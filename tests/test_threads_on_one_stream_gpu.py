"""Several threads that call on one stream: a planned call is two or three launches, which hand the plan on through
scratch memory that belongs to the stream, and a divided call puts its parts there."""
import os
import subprocess
import sys
import threading

import pytest
import torch

import fused_attention_b200 as fa

pytestmark = pytest.mark.gpu


def _call(B, R, L, H, kind, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    q, k, v = (torch.randn(B, L, R * H, generator=g, device="cuda").half() for _ in range(3))
    mask = None
    if kind == "causal":
        mask = torch.triu(torch.full((L, L), float("-inf"), device="cuda", dtype=torch.float16), diagonal=1).repeat(B, 1, 1)
    elif kind == "padding":
        mask = torch.zeros(B, L, L, device="cuda", dtype=torch.float16)
        for b in range(B):
            mask[b, :, L * (b + 1) // (B + 1):] = float("-inf")
    elif kind == "dense":
        mask = torch.randn(B, L, L, generator=g, device="cuda").half()
    return lambda: fa.attention_forward(H, 32, q, k, v, mask)


# aligned masks (two launches behind the plan), unaligned ones (their copy is in the scratch), divided calls without a mask
@pytest.mark.parametrize("kinds", [
    [(2, 20, 1021, 64, "causal"), (3, 8, 1021, 64, "dense"), (2, 20, 905, 64, "padding"), (1, 4, 3000, 128, None)],
    [(2, 30, 2048, 64, "causal"), (2, 30, 2048, 64, "padding"), (2, 30, 2048, 64, "dense"), (1, 8, 2500, 64, None)],
    [(4, 16, 2048, 128, "causal"), (2, 20, 1101, 128, "padding"), (1, 3, 4096, 128, None), (2, 30, 2048, 32, "causal")]])
def test_results_do_not_depend_on_the_other_threads_of_the_stream(kinds):
    calls = [_call(*kind, seed) for seed, kind in enumerate(kinds)]
    alone = []
    for call in calls:
        alone.append(call())
        torch.cuda.synchronize()
    wrong = []
    gate = threading.Barrier(len(calls))

    def work(i):
        try:
            for _ in range(8):
                gate.wait(60)
                outs = [calls[i]() for _ in range(6)]
                torch.cuda.synchronize()
                wrong.extend(i for y in outs if not torch.equal(alone[i], y))
        except Exception as exc:  # noqa: BLE001
            wrong.append((i, exc))

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(calls))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert wrong == []
    assert fa.read_status(0) == (0, 0)


PER_THREAD = """
import threading, torch, fused_attention_b200 as fa
from fused_attention_b200 import _lib
from fused_attention_b200.workloads import make_inputs
B, R, L, H = 1, 4, 3000, 128
lib = _lib.load()
def call(x, y, stream):
    _lib.check(lib.fa_b200_attention_forward(x[0].data_ptr(), x[1].data_ptr(), x[2].data_ptr(), None, y.data_ptr(),
                                             B, L, R * H, H, 0, 0, stream, 0))
xs = [[t.cuda() for t in make_inputs(B, L, R * H, 1.0, seed)] for seed in range(3)]
ys = [[torch.empty_like(xs[0][0]) for _ in range(30)] for _ in xs]
alone = [torch.empty_like(xs[0][0]) for _ in xs]
for x, y in zip(xs, alone):
    call(x, y, 0)
torch.cuda.synchronize()
def work(i):
    for y in ys[i]:
        call(xs[i], y, 2)            # cudaStreamPerThread
threads = [threading.Thread(target=work, args=(i,)) for i in range(3)]
for t in threads: t.start()
for t in threads: t.join()
torch.cuda.synchronize()
assert all(torch.equal(alone[i], y) for i in range(3) for y in ys[i])
assert fa.read_status(0) == (0, 0)
"""


def test_the_per_thread_stream_is_another_stream_in_every_thread():
    """One handle, a stream per thread: divided calls of three threads do not share scratch (a process of its own, where
    the four buffers are free)."""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    subprocess.run([sys.executable, "-c", PER_THREAD], check=True, cwd=root, timeout=300)
