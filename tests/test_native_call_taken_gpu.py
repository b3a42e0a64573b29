"""What the extension module's call takes itself, and what it passes back to Python's checks."""
import os

import numpy as np
import pytest
import torch

import fused_attention_b200 as fa
from fused_attention_b200 import _lib, api, build
from test_native_call_gpu import Counting, Tagged, inputs

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not os.path.exists(build.ext_path()), reason="extension module not built")]


@pytest.fixture(scope="module")
def native():
    call = api._load_native()
    return lambda *args: call(_lib.load().forward_entry, *args)


@pytest.mark.parametrize("masked", [False, True])
def test_plain_calls_are_taken(native, masked):
    q, k, v, m = inputs(masked=masked)
    expected = fa.attention_forward(32, 32, q, k, v, m, flags=_lib.FLAG_SYNC)
    assert torch.equal(native(32, 32, q, k, v, m, _lib.FLAG_SYNC), expected)
    with torch.cuda.stream(torch.cuda.Stream()):
        assert torch.equal(native(32, 32, q, k, v, m, _lib.FLAG_SYNC), expected)
    y = native(32, 32, q.clone().requires_grad_(), k, v, m, _lib.FLAG_SYNC)
    assert torch.equal(y, expected) and not y.requires_grad


def test_a_failed_call_gives_its_status(native):
    q, k, v, _ = inputs()
    assert native(32, 32, q, k, v, None, 1 << 20) == _lib.ERR_FLAGS


def test_everything_else_is_passed_back(native):
    q, k, v, m = inputs()
    strided = k.transpose(0, 1).contiguous().transpose(0, 1)
    for args in ((np.int64(32), 32, q, k, v, m, 0), (32, 32, q.as_subclass(Tagged), k, v, m, 0), (48, 32, q, k, v, m, 0),
                 (32, 128, q, k, v, m, 0), (64, 32, q, k, v, m, 0), (32, 32, q.float(), k, v, m, 0), (32, 32, q.cpu(), k, v, m, 0),
                 (32, 32, q, strided, v, m, 0), (32, 32, q, k, v[0], m, 0), (32, 32, q, k, v[:, 1:].contiguous(), m, 0),
                 (32, 32, q, k, v, m[:, 1:].contiguous(), 0), (32, 32, q, k, v, m, -1), (32, 32, q, k, v, m, 1 << 32),
                 (32, 32, None, k, v, m, 0), (32, 32, q, k, v, 0, 0), (32, 32, q, k, v, m, 0.0)):
        assert native(*args) is None


def test_a_function_mode_sees_the_call(native):
    q, k, v, m = inputs()
    fa.attention_forward(32, 32, q, k, v, m)
    Counting.calls = 0
    with Counting():
        assert native(32, 32, q, k, v, m, 0) is None and Counting.calls == 0
        fa.attention_forward(32, 32, q, k, v, m)
    assert Counting.calls > 0
