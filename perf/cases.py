"""The attention calls that are timed: what a user of this operator has it do, through its public entry points.

A case is one call ``Y = softmax(Q K^T / sqrt(H) + mask) V`` on fp16 ``[B, L, R*H]`` tensors:

  entry   "package"    fused_attention_b200.attention_forward (Python mirror of the operator)
          "extension"  fused_attn.attention_forward, the drop-in torch extension module
          "host"       fused_attention_b200.attention_forward_host on pinned host tensors
  B R L H batch, heads, sequence length, head dimension;  sigma: standard deviation of Q, K and V
  mask    "none", or an additive fp16 [B, L, L] mask:
          "causal"     -inf above the diagonal, 0 elsewhere
          "padding"    every batch entry has a length of its own; -inf at the keys beyond it
          "bias"       a dense finite bias (relative positions), N(0, 1)
"""
import importlib.util
import math
import os

import torch

import fused_attention_b200 as fa

MASKS = ("none", "causal", "padding", "bias")


def listed():
    return [
        # the smallest call in use: a few heads of a short sequence, where the launch and the host side are the time
        dict(name="tiny", entry="package", B=1, R=4, L=256, H=64, sigma=1.0, mask="none"),
        # encoder layer at batch 8, every sequence full
        dict(name="bert_base", entry="extension", B=8, R=12, L=512, H=64, sigma=1.0, mask="none"),
        # the same layer on a batch of sequences of different lengths, padded to 512
        dict(name="bert_padded", entry="extension", B=8, R=12, L=512, H=64, sigma=1.0, mask="padding"),
        # image encoder: 196 patches and a class token, a ragged length
        dict(name="vit_l16_ragged", entry="package", B=64, R=16, L=197, H=64, sigma=1.0, mask="none"),
        # attention inside 7x7 windows of an image with a bias per position: many short problems, unaligned mask rows
        dict(name="window_bias", entry="package", B=256, R=8, L=49, H=32, sigma=1.0, mask="bias"),
        # small heads over a long sequence
        dict(name="small_heads", entry="package", B=8, R=16, L=1024, H=32, sigma=1.0, mask="none"),
        # decoder prompts of an odd length: causal, mask rows on no 16-byte boundary
        dict(name="causal_odd", entry="extension", B=4, R=12, L=1021, H=64, sigma=1.0, mask="causal"),
        # prefill of a large decoder, the headline shape, and the same with the causal mask it has in use
        dict(name="llama7b_prefill", entry="package", B=4, R=32, L=2048, H=128, sigma=0.5, mask="none"),
        dict(name="llama7b_causal", entry="package", B=4, R=32, L=2048, H=128, sigma=0.5, mask="causal"),
        # one sequence, the few heads that a tensor-parallel rank holds, a ragged length: fewer work items than SMs
        dict(name="few_heads", entry="extension", B=1, R=4, L=3000, H=128, sigma=1.0, mask="none"),
        # long context, the largest call
        dict(name="long_context", entry="package", B=1, R=32, L=16384, H=128, sigma=1.0, mask="none"),
        # a program that holds its tensors in host memory
        dict(name="host_buffers", entry="host", B=2, R=32, L=1024, H=128, sigma=0.5, mask="none"),
    ]


def _log_int(rng, low, high):
    return max(low, min(high, round(math.exp(rng.uniform(math.log(low), math.log(high + 1))))))


def draw(rng):
    """One more call of the same kinds; a length is a multiple of 128, of 8 or odd with the same likelihood."""
    kind = rng.choice(("encoder", "image", "window", "small_heads", "decoder", "prefill", "few_heads", "long", "host"))
    H, sigma, mask, entry = 64, 1.0, "none", rng.choice(("package", "extension"))
    if kind == "encoder":
        B, R, L, mask = _log_int(rng, 1, 32), rng.choice((4, 8, 12, 16)), _log_int(rng, 64, 1024), rng.choice(("none", "padding"))
    elif kind == "image":
        B, R, L = _log_int(rng, 8, 128), rng.choice((6, 12, 16)), rng.choice((7, 12, 14, 16, 24)) ** 2 + 1
    elif kind == "window":
        H, B, R = rng.choice((16, 32)), _log_int(rng, 64, 1024), rng.choice((3, 4, 6, 8, 16))
        L, mask = rng.randint(4, 12) ** 2, rng.choice(("none", "bias", "bias"))
    elif kind == "small_heads":
        H, B, R, L = rng.choice((16, 32)), _log_int(rng, 1, 16), rng.choice((4, 8, 16)), _log_int(rng, 128, 2048)
        mask = rng.choice(MASKS)
    elif kind == "decoder":
        H, B, R, L = rng.choice((64, 128)), _log_int(rng, 1, 8), rng.choice((8, 12, 16, 32)), _log_int(rng, 100, 2048)
        mask = "causal"
    elif kind == "prefill":
        H, B, R, L, sigma = 128, _log_int(rng, 1, 4), rng.choice((16, 32, 40)), _log_int(rng, 256, 4096), 0.5
        mask = rng.choice(("none", "causal"))
    elif kind == "few_heads":
        H, B, R, L = rng.choice((64, 128)), 1, rng.randint(1, 8), _log_int(rng, 512, 8192)
    elif kind == "long":
        H, B, R, L = 128, 1, rng.choice((4, 8, 16, 32)), _log_int(rng, 4096, 16384)
    else:
        H, B, R, L, sigma, entry = rng.choice((64, 128)), _log_int(rng, 1, 4), rng.choice((8, 16, 32)), _log_int(rng, 256, 1024), 0.5, "host"
    if kind not in ("image", "window"):
        step = rng.choice((128, 8, 1))
        L = max(step, L // step * step)
        if step == 1 and L % 2 == 0:
            L -= 1
    return dict(entry=entry, B=B, R=R, L=L, H=H, sigma=sigma, mask=mask)


def _lengths(B, L, seed):
    """Lengths of the entries of a padded batch: spread evenly from a quarter of L to all of it, in an order of the seed."""
    even = [max(1, round(L * (0.25 + 0.75 * (b + 1) / B))) for b in range(B)]
    order = torch.randperm(B, generator=torch.Generator().manual_seed(seed)).tolist()
    return [even[i] for i in order]


def _mask(case, seed, g):
    B, L = case["B"], case["L"]
    if case["mask"] == "none":
        return None
    if case["mask"] == "bias":
        return torch.randn(B, L, L, generator=g, device="cuda", dtype=torch.float16)
    if case["mask"] == "causal":
        one = torch.full((L, L), float("-inf"), device="cuda", dtype=torch.float16).triu(1)
        return one.unsqueeze(0).repeat(B, 1, 1)
    keys = torch.arange(L, device="cuda")
    beyond = keys[None, :] >= torch.tensor(_lengths(B, L, seed), device="cuda")[:, None]
    row = torch.zeros(B, L, device="cuda", dtype=torch.float16).masked_fill_(beyond, float("-inf"))
    return row.unsqueeze(1).repeat(1, L, 1)


def _extension():
    """The torch extension module `fused_attn`, from where the build of this package puts it."""
    from fused_attention_b200.build import ext_path
    spec = importlib.util.spec_from_file_location("fused_attn", os.path.abspath(ext_path()))
    module = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(module)
    return module


def _inputs(case, seed):
    """Q, K, V and the mask (or None) of a case, on the GPU."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    shape = (case["B"], case["L"], case["R"] * case["H"])
    q, k, v = (torch.randn(shape, generator=g, device="cuda", dtype=torch.float16) * case["sigma"] for _ in range(3))
    return q, k, v, _mask(case, seed, g)


def prepare(case, seed):
    B, L, F = case["B"], case["L"], case["R"] * case["H"]
    q, k, v, mask = _inputs(case, seed)
    chunk = 64 if case["H"] >= 32 else 32
    s = dict(entry=case["entry"], H=case["H"], chunk=chunk, q=q, k=k, v=v, mask=mask)
    if case["entry"] == "extension":
        s["call"] = _extension().attention_forward
    elif case["entry"] == "host":
        for name in "qkv":
            s[name] = s[name].cpu().pin_memory()
        s["out"] = torch.empty(B, L, F, dtype=torch.float16).pin_memory()
    return s


def run(state):
    s = state
    if s["entry"] == "host":
        return fa.attention_forward_host(s["H"], s["chunk"], s["q"], s["k"], s["v"], s["mask"], out=s["out"])
    call = s["call"] if s["entry"] == "extension" else fa.attention_forward
    return call(s["H"], s["chunk"], s["q"], s["k"], s["v"], s["mask"])


def work(case):
    """Q, K, V and the mask read once and Y written once; two products of H multiply-adds for every pair of a query
    and a key that the mask leaves in."""
    B, R, L, H = (case[n] for n in "BRLH")
    pairs = B * L * L
    if case["mask"] == "causal":
        pairs = B * L * (L + 1) // 2
    elif case["mask"] == "padding":
        pairs = L * sum(_lengths(B, L, 0))
    masked = 0 if case["mask"] == "none" else 2 * B * L * L
    return {"bytes": 8 * B * L * R * H + masked, "flops": 4 * pairs * R * H}


def tolerance(case):
    """fp16 results of fp16 operands, P rounded to fp16 once and everything else in fp32: measured against attention in
    64 (the largest calls 32) bits the results are off by 2.4e-4 to 3.0e-4 (rounding Y to fp16 alone: 2.0e-4), and no
    value by more than 5.5e-3, over the listed and fourteen drawn cases; four times that."""
    return {"rel": 1.2e-3, "max": 2.2e-2}


def exact(case, seed):
    """The same result in 64 bits: one batch entry and head, and at most 2048 of its queries, at a time."""
    H = case["H"]
    q, k, v, mask = _inputs(case, seed)
    y = torch.empty(q.shape, dtype=torch.float64, device=q.device)
    for b in range(case["B"]):
        for c in range(0, q.shape[2], H):
            kd, vd = k[b, :, c:c + H].double(), v[b, :, c:c + H].double()
            for i in range(0, case["L"], 2048):
                s = q[b, i:i + 2048, c:c + H].double() @ kd.T / math.sqrt(H)
                if mask is not None:
                    s += mask[b, i:i + 2048].double()
                y[b, i:i + 2048, c:c + H] = torch.softmax(s, dim=-1) @ vd
    return y.cpu() if case["entry"] == "host" else y
