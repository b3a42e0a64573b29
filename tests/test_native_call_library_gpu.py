"""attention_forward calls the library that the package has loaded, also where that is not the one the extension module links."""
import os

import pytest
import torch

import fused_attention_b200 as fa
from fused_attention_b200 import _lib, build

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("variant", [build.DEBUG_LIB, build.CYCLES_LIB], ids=["checked", "clock counting"])
def test_calls_go_to_the_loaded_library(monkeypatch, variant):
    if not os.path.exists(variant):
        pytest.skip(f"{os.path.basename(variant)} not built")
    B, L, H, R = 2, 2048, 64, 30
    q, k, v = (torch.randn(B, L, R * H, device="cuda", dtype=torch.float16) for _ in range(3))
    dense = torch.randn(B, L, L, device="cuda", dtype=torch.float16)
    causal = torch.full((L, L), float("-inf"), dtype=torch.float16, device="cuda").triu(1).repeat(B, 1, 1)
    expected = fa.attention_forward(H, 64, q, k, v, causal, flags=_lib.FLAG_SYNC)
    monkeypatch.setattr(_lib, "_lib", None)
    monkeypatch.setattr(_lib, "LIB_PATH", variant)
    launch, _ = fa.bind_forward(H, 64, q, k, v, dense)
    launch()                                           # (through ctypes)
    assert fa.plan_taken() is False
    y = fa.attention_forward(H, 64, q, k, v, causal, flags=_lib.FLAG_SYNC)
    assert fa.plan_taken() is True and torch.equal(y, expected)
    assert fa.read_status(0) == (0, 0)
