"""The host-pointer GEMV with x in page-locked memory: the CTAs of a launch stage x together, counted by a device counter
that outlives the call."""
from __future__ import annotations

import ctypes as C
import os
import subprocess
import sys

import numpy as np
import pytest

from tensormark_b200 import lib, synth
from tests.gpu_util import dev_bytes, dev_f32, gemv_dev, ptr

pytestmark = pytest.mark.gpu


def pinned(torch, a: np.ndarray):
    return torch.from_numpy(a).pin_memory()


def check_call(cuda, torch, orc, dt, n, k, seed):
    W, x = synth.make_weights(dt, n, k, seed=seed), synth.make_activations(k, seed=seed + 1)
    xp, yp = pinned(torch, x), torch.full((n,), float("nan")).pin_memory()
    lib.check(cuda.tm_cuda_gemv_q(ptr(xp), W.ctypes.data, ptr(yp), n, k, dt), "tm_cuda_gemv_q")
    cuda.tm_cuda_release_weights()
    y64, yabs = orc.gemv_f64(dt, W, x, n, k)
    assert np.all(np.abs(yp.numpy() - y64) <= 1e-4 * yabs), (dt, n, k)
    return yp.numpy().copy()


def test_cta_that_does_not_wait_for_the_others(cuda, torch_mod, orc):
    """A CTA that has waited long enough stages x for itself, with the same bits: here one whose patience is nil, in a child."""
    shapes = [(synth.Q4_0, 256, 2048), (synth.Q8_0, 40, 14336), (synth.Q6_K, 3000, 2048)]
    want = [check_call(cuda, torch_mod, orc, dt, n, k, seed=30) for dt, n, k in shapes]
    code = ("import numpy as np, torch\n"
            "from oracle import binding\n"
            "from tensormark_b200 import lib\n"
            "from tests.test_gpu_host_gemv import check_call\n"
            "L = lib.load()\n"
            "lib.check(L.tm_cuda_init(-1), 'tm_cuda_init')\n"
            f"for dt, n, k in {shapes}:\n"
            "    print(check_call(L, torch, binding.oracle(), dt, n, k, seed=30).tobytes().hex())\n")
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", code], cwd=root, env=dict(os.environ, TM_GEMV_SHARE_WAIT_US="0"), capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr
    for line, w in zip(r.stdout.split(), want, strict=True):
        assert np.array_equal(np.frombuffer(bytes.fromhex(line), np.float32), w)


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


def test_calls_in_a_row(cuda, torch_mod, orc):
    """One process, page-locked x and y: formats, fewer and more groups of x than CTAs, a K that is no multiple of 256, a
    scratch buffer that grows and is then larger than needed, x changed between two calls, pageable calls in between. Bits are
    those of the entry with device pointers."""
    torch = torch_mod
    shapes = [(synth.Q4_0, 256, 2048), (synth.Q8_0, 1, 14336), (synth.Q4_1, 40, 14336), (synth.Q4_1, 5632, 2176), (synth.Q6_K, 300, 2048),
              (synth.Q4_0, 17, 256), (synth.GGUF_Q4_0, 9000, 4096), (synth.Q5_K, 7, 14336), (synth.Q4_0, 130, 352), (synth.Q4_K, 148, 512), (synth.Q8_0, 20, 28672),
              (synth.Q4_0, 9, 33024)]
    keep = []                                    # copies on the device go by host address
    for i, (dt, n, k) in enumerate(shapes):
        W = synth.make_weights(dt, n, k, seed=40 + i)
        keep.append(W)
        Wd = dev_bytes(torch, W)
        xp, yp = pinned(torch, np.empty(k, np.float32)), torch.empty(n).pin_memory()
        for again in range(3):
            x = synth.make_activations(k, seed=60 + 10 * i + again)
            want = gemv_dev(cuda, torch, dt, Wd, dev_f32(torch, x), n, k)
            xp.copy_(torch.from_numpy(x))
            yp.fill_(float("nan"))
            lib.check(cuda.tm_cuda_gemv_q(ptr(xp), W.ctypes.data, ptr(yp), n, k, dt), "tm_cuda_gemv_q")
            assert np.array_equal(yp.numpy(), want), (dt, n, k)
            if again == 1:
                y = np.empty(n, np.float32)
                lib.check(cuda.tm_cuda_gemv_q(x.ctypes.data, W.ctypes.data, y.ctypes.data, n, k, dt), "tm_cuda_gemv_q")
                assert np.array_equal(y, want)
        y64, yabs = orc.gemv_f64(dt, W, x, n, k)
        assert np.all(np.abs(want - y64) <= 1e-4 * yabs), (dt, n, k)
