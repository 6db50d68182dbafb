"""The host-pointer GEMV with x in page-locked memory: the CTAs of a launch stage x together, counted by a device counter
that outlives the call."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from tensormark_b200 import lib, synth
from tests.gpu_util import ptr

pytestmark = pytest.mark.gpu


def pinned(torch, a: np.ndarray):
    return torch.from_numpy(a).pin_memory()


def test_call_that_never_ran(cuda, torch_mod, orc):
    """A call inside a capture is refused when it comes to wait, and its kernel never runs: the next call must not wait for it."""
    torch = torch_mod
    n, k, dt = 300, 2048, synth.Q4_0
    W, x = synth.make_weights(dt, n, k, seed=20), synth.make_activations(k, seed=21)
    xp, yp = pinned(torch, x), torch.empty(n).pin_memory()
    call = lambda: cuda.tm_cuda_gemv_q(ptr(xp), W.ctypes.data, ptr(yp), n, k, dt)  # noqa: E731
    lib.check(call(), "tm_cuda_gemv_q")
    want = yp.numpy().copy()
    assert cuda.tm_cuda_tok_graph_begin(), lib.last_error()
    refused = not call()
    assert cuda.tm_cuda_tok_graph_end() < 0 and refused
    yp.zero_()
    lib.check(call(), "tm_cuda_gemv_q")
    assert np.array_equal(yp.numpy(), want)
    y64, yabs = orc.gemv_f64(dt, W, x, n, k)
    assert np.all(np.abs(want - y64) <= 1e-4 * yabs)
