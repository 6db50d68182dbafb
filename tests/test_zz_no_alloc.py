"""The allocation-free decode attention entry against the ordinary one.

Collected last on purpose (file name): if it fails, a run that stops at the first failure has
already executed every other test. The entry under test keeps its split-K scratch in a static
device array, for hosts that have no device memory left to allocate from or cannot afford an
allocation on their token path; it must give what tm_cuda_attn_decode_dev gives, call after call,
although both calls write the same array."""
from __future__ import annotations

import os
import subprocess
import sys

import numpy as np
import pytest

from tensormark_b200 import lib
from tests.gpu_util import ptr, stream_ptr

pytestmark = pytest.mark.gpu


def _case(torch, Hn, KVH, dh, ctx, seed, half, off=0):
    """q, K, V; off: elements that the caches lie behind a 16-byte boundary."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    q = torch.randn(Hn * dh, generator=g, device="cuda", dtype=torch.float32)
    k = torch.randn(KVH * ctx * dh + 8, generator=g, device="cuda", dtype=torch.float32)
    v = torch.randn(KVH * ctx * dh + 8, generator=g, device="cuda", dtype=torch.float32)
    if half:
        k, v = k.half(), v.half()
    return q, k[off:], v[off:]


@pytest.mark.parametrize("half", [1, 0])
def test_static_scratch_attention_matches_call_after_call(cuda, torch_mod, half):
    """Calls in a row share the array, and only the form of two launches uses it: a long call, a shorter one with as many splits
    (18), one with four (caches off the 16-byte grid are merged by a second launch at any length), one in a single launch, and
    again a long one."""
    torch = torch_mod
    Hn, KVH, dh, ctx = 32, 8, 128, 1024          # the decode-chain head geometry
    scale = 1.0 / np.sqrt(dh)
    sp = stream_ptr(torch)
    for call, (allow, off, launches) in enumerate([(1000, 0, 2), (640, 0, 2), (97, 1, 2), (97, 0, 1), (1024, 0, 2)]):
        q, k, v = _case(torch, Hn, KVH, dh, ctx, 20 + call, half, off)
        need = cuda.tm_cuda_attn_decode_scratch(Hn, KVH, dh, ctx, allow)
        scratch = torch.empty(need // 4 + 4, dtype=torch.float32, device="cuda")
        want = torch.empty(Hn * dh, dtype=torch.float32, device="cuda")
        got = torch.full((Hn * dh,), float("nan"), dtype=torch.float32, device="cuda")
        lib.check(cuda.tm_cuda_attn_decode_dev(ptr(q), ptr(k), ptr(v), ptr(scratch), need, ptr(want), Hn, KVH, dh, ctx,
                                               allow, scale, half, sp), "tm_cuda_attn_decode_dev")
        before, launched = torch.cuda.memory_allocated(), cuda.tm_cuda_launch_count()
        lib.check(cuda.tm_cuda_attn_decode_static_dev(ptr(q), ptr(k), ptr(v), ptr(got), Hn, KVH, dh, ctx, allow, scale,
                                                      half, sp), "tm_cuda_attn_decode_static_dev")
        torch.cuda.synchronize()
        assert torch.cuda.memory_allocated() == before
        assert cuda.tm_cuda_launch_count() - launched == launches
        # the tolerance the attention parity tests use (1e-3 relative, 2e-5 absolute)
        assert np.allclose(got.cpu().numpy(), want.cpu().numpy(), rtol=1e-3, atol=2e-5)


ALONE = """
import ctypes as C
import torch
from tensormark_b200 import lib
L = lib.load()
torch.cuda.set_device(0)
st = C.c_void_p(torch.cuda.current_stream().cuda_stream)
P = lambda t: C.c_void_p(t.data_ptr())
H, KVH, dh, ctx, scale = 32, 8, 128, 1024, 128 ** -0.5
g = torch.Generator(device="cuda").manual_seed(5)
q = torch.randn(H, dh, generator=g, device="cuda")
k, v = (torch.randn(KVH, ctx, dh, generator=g, device="cuda").half() for _ in range(2))
for allow, launches in ((300, 1), (1000, 2)):
    out = torch.full((H, dh), float("nan"), device="cuda")
    before = L.tm_cuda_launch_count()
    assert L.tm_cuda_attn_decode_static_dev(P(q), P(k), P(v), P(out), H, KVH, dh, ctx, allow, scale, 1, st), lib.last_error()
    torch.cuda.synchronize()
    assert L.tm_cuda_launch_count() - before == launches, (allow, L.tm_cuda_launch_count() - before)
    s = torch.einsum("grd,gpd->grp", q.double().view(KVH, H // KVH, dh), k[:, :allow].double()) * scale
    want = torch.einsum("grp,gpd->grd", s.softmax(-1), v[:, :allow].double()).reshape(H, dh)
    assert torch.allclose(out.double(), want, rtol=1e-3, atol=2e-5), (out - want).abs().max()
"""


def test_static_entry_alone_in_a_process(cuda):
    """A host that calls nothing else: the library is not initialised, and the entry still takes the launches that the SMs of
    the current device call for."""
    r = subprocess.run([sys.executable, "-c", ALONE], cwd=os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]


def test_static_scratch_refuses_what_does_not_fit(cuda, torch_mod):
    torch = torch_mod
    Hn, KVH, dh, ctx, allow = 64, 8, 128, 1024, 1024      # 19 splits x 64 heads x 130 floats = 632 KB > 512 KB
    q, k, v = _case(torch, Hn, KVH, dh, ctx, 3, 1)
    out = torch.zeros(Hn * dh, dtype=torch.float32, device="cuda")
    before = cuda.tm_cuda_fallback_count()
    assert not cuda.tm_cuda_attn_decode_static_dev(ptr(q), ptr(k), ptr(v), ptr(out), Hn, KVH, dh, ctx, allow, 0.1, 1,
                                                   stream_ptr(torch))
    assert cuda.tm_cuda_fallback_count() == before + 1
    assert "static array holds" in lib.last_error()
    torch.cuda.synchronize()
    assert not out.any()                                   # nothing ran
