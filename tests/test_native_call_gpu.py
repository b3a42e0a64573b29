"""attention_forward in native code and through ctypes: the same results, and the same errors, for every kind of argument."""
import numpy as np
import pytest
import torch
from torch.overrides import TorchFunctionMode

import fused_attention_b200 as fa
from fused_attention_b200 import _lib, api

pytestmark = pytest.mark.gpu


class Tagged(torch.Tensor):
    pass


class Counting(TorchFunctionMode):
    calls = 0

    def __torch_function__(self, func, types, args=(), kwargs=None):
        Counting.calls += 1
        return func(*args, **(kwargs or {}))


def inputs(B=2, L=130, R=3, H=32, masked=True):
    g = torch.Generator(device="cuda").manual_seed(5)
    q, k, v = (torch.randn(B, L, R * H, generator=g, device="cuda", dtype=torch.float16) for _ in range(3))
    return q, k, v, torch.randn(B, L, L, generator=g, device="cuda", dtype=torch.float16) if masked else None


def both(monkeypatch, call):
    with monkeypatch.context() as m:
        m.setattr(api, "_native", lambda *args: None)
        expected = call()
    return call(), expected


@pytest.mark.parametrize("masked", [False, True])
@pytest.mark.parametrize("kind", ["plain", "needs_grad", "subclass", "mode", "numpy_int", "other_stream"])
def test_native_and_ctypes_agree(monkeypatch, kind, masked):
    q, k, v, m = inputs(masked=masked)
    H = np.int64(32) if kind == "numpy_int" else 32
    if kind == "needs_grad":
        q.requires_grad_()
    if kind == "subclass":
        q = q.as_subclass(Tagged)

    def call():
        if kind == "mode":
            with Counting():
                return fa.attention_forward(H, 32, q, k, v, m, flags=_lib.FLAG_SYNC)
        if kind == "other_stream":
            with torch.cuda.stream(torch.cuda.Stream()):
                return fa.attention_forward(H, 32, q, k, v, m, flags=_lib.FLAG_SYNC)
        return fa.attention_forward(H, 32, q, k, v, m, flags=_lib.FLAG_SYNC)
    y, expected = both(monkeypatch, call)
    assert type(y) is type(expected) and not y.requires_grad and not expected.requires_grad and torch.equal(y, expected)
    assert kind != "mode" or Counting.calls > 0


@pytest.mark.parametrize("spoil", [
    dict(head_dim=48), dict(head_dim=-32), dict(chunk=128), dict(chunk=24), dict(q="float"), dict(q="cpu"), dict(k="strided"),
    dict(v="rank"), dict(v="shape"), dict(mask="shape"), dict(mask="float"), dict(head_dim=64), dict(flags=1 << 20),
    dict(q="none")])
def test_what_is_refused_is_refused_alike(monkeypatch, spoil):
    q, k, v, m = inputs()
    change = {"float": lambda t: t.float(), "cpu": lambda t: t.cpu(), "strided": lambda t: t.transpose(0, 1).contiguous().transpose(0, 1),
              "rank": lambda t: t[0], "shape": lambda t: t[:, 1:].contiguous(), "none": lambda t: None}
    args = {n: (change[spoil[n]](t) if n in spoil else t) for n, t in dict(q=q, k=k, v=v, mask=m).items()}

    def call():
        try:
            fa.attention_forward(spoil.get("head_dim", 32), spoil.get("chunk", 32), args["q"], args["k"], args["v"], args["mask"],
                                 flags=spoil.get("flags", 0))
        except Exception as e:
            return type(e), str(e)
    y, expected = both(monkeypatch, call)
    assert expected is not None and y == expected
