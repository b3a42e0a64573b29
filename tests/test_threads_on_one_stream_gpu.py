"""Several threads that call on one stream: a planned call is two or three launches, which hand the plan on through
scratch memory that belongs to the stream, and a divided call puts its parts there."""
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
