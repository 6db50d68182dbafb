"""The lane's GEMV with its transforms of x (RMSNorm, SiLU * up) and the residual add, over the kernels that serve it: rows
on the 16-byte grid, rows off it, rows on odd addresses, x staged by the CTAs and by a launch of its own."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from tensormark_b200 import lib, synth
from tests.bounds import activation_rounding_bound

pytestmark = pytest.mark.gpu

XS, US, YS = 95, 96, 97          # slots of this test only
EPS = 1e-5
_KEEP = []                       # registrations and norm weights go by host address


def up(cuda, slot, a):
    lib.check(cuda.tm_cuda_tok_upload(slot, 0, a.ctypes.data, a.nbytes), "tok_upload")


def fused(cuda, orc, dt, n, k, shift, op, accumulate, x, W=None):
    rng = np.random.default_rng(k + op)
    W = synth.make_weights(dt, n, k, seed=91) if W is None else W
    blob = np.zeros(W.size + shift + 32, np.uint8)
    blob[shift:shift + W.size] = W.reshape(-1)
    u = (1 + 0.1 * rng.standard_normal(k)).astype(np.float32)
    y0 = rng.standard_normal(n).astype(np.float32)
    _KEEP.extend((blob, u))
    woff = C.c_uint64(0)
    wid = cuda.tm_cuda_tok_wbuf(blob.ctypes.data, blob.nbytes, None, 0, 0, C.byref(woff))
    assert wid >= 1000, lib.last_error()
    for slot, a in ((XS, x), (US, u), (YS, y0)):
        up(cuda, slot, a)
    rows, off = (C.c_uint * 1)(n), (C.c_uint64 * 1)(woff.value + shift)
    assert cuda.tm_cuda_tok_begin(), lib.last_error()
    cuda.tm_cuda_tok_gemv_fused(XS, 0, op, US, 0, C.c_void_p(u.ctypes.data) if op == 1 else None, EPS, wid, YS, 0, n, k, dt, off, rows, 1, accumulate)
    assert cuda.tm_cuda_tok_flush(), lib.last_error()
    y = np.empty(n, np.float32)
    lib.check(cuda.tm_cuda_tok_download(YS, 0, y.ctypes.data, y.nbytes), "tok_download")
    x64, u64 = x.astype(np.float64), u.astype(np.float64)
    t = x64 if op == 0 else x64 / np.sqrt(np.mean(x64 * x64) + EPS) * u64 if op == 1 else x64 / (1 + np.exp(-x64)) * u64
    wd = orc.dequant(dt, W, n * k).reshape(n, k).astype(np.float64)
    base = y0.astype(np.float64) if accumulate else 0.0
    yabs = np.abs(wd) @ np.abs(t)
    # the residual add rounds once more
    err = np.maximum(np.abs(y - (wd @ t + base)) - 6e-8 * np.abs(base + wd @ t), 0.0)
    return err, yabs, W, t.astype(np.float32)


@pytest.mark.parametrize("accumulate", [0, 1])
@pytest.mark.parametrize("op", [0, 1, 2])
@pytest.mark.parametrize("dt,n,k,shift", [
    (synth.Q4_0, 300, 2048, 0), (synth.Q8_0, 40, 14336, 0), (synth.Q6_K, 149, 4096, 0),
    (synth.Q4_0, 300, 2080, 0), (synth.Q8_0, 77, 4128, 0), (synth.Q4_1, 50, 14368, 0), (synth.Q6_K, 149, 2816, 0), (synth.Q5_K, 33, 2048, 2),
    (synth.Q4_0, 30, 2048, 7), (synth.Q8_0, 30, 2048, 7), (synth.Q4_1, 30, 2048, 7), (synth.Q5_K, 30, 2048, 7), (synth.Q6_K, 30, 2048, 7),
    (synth.Q4_K, 30, 2048, 7), (synth.GGUF_Q4_0, 30, 2048, 7), (synth.TQ2, 30, 2048, 0),
])
def test_transforms(cuda, orc, dt, n, k, shift, op, accumulate):
    x = synth.make_activations(k, seed=92)
    err, yabs, W, t = fused(cuda, orc, dt, n, k, shift, op, accumulate, x)
    planes = dt != synth.TQ2 and W.shape[1] % 16 == 0 and shift == 0        # two planes of x; everywhere else x is fp32, or as close
    bound = activation_rounding_bound(orc, dt, W, t, n, k) if planes else 0.0
    assert np.all(err <= bound + 2e-6 * yabs), float((err / yabs).max())


def test_gate_far_below_zero(cuda, orc):
    """Rows off the grid keep x to fp32's last bits, so the gate has to be as good: one activation per row, where the gate is
    e^x. expf 2 ulp, the sum, the quotient and the product half an ulp each, the planes and the scale a quarter: 4 x 2^-23."""
    n, k = 129, 4128
    x = np.linspace(-19, -9, k).astype(np.float32)
    one = np.zeros((n, k // 32, 34), np.uint8)
    one[:, :, 0:2] = np.full(1, 1.0, np.float16).view(np.uint8)
    pick = np.arange(n) * 32 + np.arange(n) % 32
    one[np.arange(n), pick // 32, 2 + pick % 32] = 1
    err, yabs, _, _ = fused(cuda, orc, synth.Q8_0, n, k, 0, 2, 0, x, W=one.reshape(n, -1))
    assert np.all(err <= 4 * 2.0 ** -23 * yabs), float((err / yabs).max())
