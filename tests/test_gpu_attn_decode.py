"""Decode attention over its whole dispatch: heads per K/V head, head dims, cache types, ranges that end inside a stage,
caches off the 16-byte grid."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from tensormark_b200 import lib
from tests.gpu_util import dev_f32, ptr, stream_ptr

pytestmark = pytest.mark.gpu


def run(cuda, torch, orc, KVH, rep, dh, ctx, allow, half, off=0, last_v=None):
    rng = np.random.default_rng(allow + rep)
    H, scale = KVH * rep, 1.0 / np.sqrt(dh)
    q = rng.standard_normal((H, dh)).astype(np.float32) * 2
    kv = rng.standard_normal((2, KVH, ctx, dh)).astype(np.float16 if half else np.float32)
    if last_v is not None:
        kv[1, :, allow - 1, ::3] = last_v
    qd = dev_f32(torch, q)
    flat = [torch.zeros(kv[0].size + 8, dtype=torch.float16 if half else torch.float32, device="cuda") for _ in range(2)]
    for t, a in zip(flat, kv):
        t[off:off + a.size] = torch.from_numpy(a.reshape(-1)).cuda()
    at = [C.c_void_p(t.data_ptr() + off * t.element_size()) for t in flat]
    need = cuda.tm_cuda_attn_decode_scratch(H, KVH, dh, ctx, allow)
    scratch = torch.empty(need // 4 + 1, dtype=torch.float32, device="cuda")
    out = torch.empty(H * dh, dtype=torch.float32, device="cuda")
    launched = cuda.tm_cuda_launch_count()
    lib.check(cuda.tm_cuda_attn_decode_dev(ptr(qd), at[0], at[1], ptr(scratch), need, ptr(out), H, KVH, dh, ctx, allow, scale,
                                           int(half), stream_ptr(torch)), "attn_decode_dev")
    launched = cuda.tm_cuda_launch_count() - launched
    torch.cuda.synchronize()
    got = out.cpu().numpy().reshape(H, dh)
    K, V = kv[0].astype(np.float32), kv[1].astype(np.float32)
    for g in range(KVH):
        want = orc.attn_group(q[g * rep:(g + 1) * rep], K[g, :allow], V[g, :allow], scale)
        assert np.allclose(got[g * rep:(g + 1) * rep], want, rtol=1e-3, atol=2e-5), (g, np.abs(got[g * rep:(g + 1) * rep] - want).max())
    return launched


@pytest.mark.parametrize("half", [False, True])
@pytest.mark.parametrize("dh", [64, 128])
@pytest.mark.parametrize("rep", [1, 2, 4, 8])
def test_heads_dims_types(cuda, torch_mod, orc, rep, dh, half):
    for allow in (1, 33, 1000):
        run(cuda, torch_mod, orc, 2, rep, dh, 1024, allow, half)


@pytest.mark.parametrize("KVH,rep,allow", [
    (148, 1, 127), (148, 1, 128), (148, 1, 129), (149, 2, 300), (37, 4, 95), (37, 4, 97), (74, 8, 57), (1, 4, 8191), (8, 4, 8192),
])
def test_ranges_around_a_stage(cuda, torch_mod, orc, KVH, rep, allow):
    run(cuda, torch_mod, orc, KVH, rep, 128, max(allow, 256), allow, True)


# launches with fp32 and with fp16 caches on 148 SMs, which hold up to seven clusters of 16 CTAs that fill an SM each
@pytest.mark.parametrize("half", [False, True])
@pytest.mark.parametrize("KVH,rep,dh,allow,launches", [
    (8, 4, 128, 3, (1, 1)), (8, 4, 128, 500, (2, 1)), (8, 4, 128, 620, (2, 2)), (4, 8, 64, 1340, (2, 1)), (4, 8, 64, 1380, (2, 2)),
    (2, 4, 64, 1150, (2, 1)), (2, 4, 64, 1500, (2, 1)), (1, 8, 64, 17, (1, 1)), (1, 8, 128, 760, (1, 1)), (1, 8, 128, 910, (2, 2)),
    (5, 4, 128, 50, (1, 1)), (3, 1, 64, 511, (1, 1)), (37, 2, 64, 300, (1, 1)), (74, 1, 128, 40, (1, 1)), (148, 1, 64, 40, (1, 1)),
    (149, 1, 64, 9, (2, 2)), (4, 4, 64, 9000, (2, 2)), (3, 4, 128, 9000, (2, 2)), (2, 2, 64, 20000, (2, 2)), (1, 8, 128, 4884, (2, 2)),
])
def test_one_launch(cuda, torch_mod, orc, KVH, rep, dh, allow, launches, half):
    """Around the lines between one launch and two: clusters of 16 down to 1, splits without a position, K/V heads that are no
    power of two or more than fit at a time; merges of 37, 49, 74 and 148 splits. The arithmetic is the same in both, and so is the
    bound; the launches say which of the two it was."""
    assert run(cuda, torch_mod, orc, KVH, rep, dh, allow + 3, allow, half) == launches[half]


@pytest.mark.parametrize("half", [False, True])
def test_caches_off_the_grid(cuda, torch_mod, orc, half):
    assert run(cuda, torch_mod, orc, 2, 4, 128, 300, 257, half, off=1) == 2
    assert run(cuda, torch_mod, orc, 3, 8, 64, 300, 300, half, off=3) == 2


@pytest.mark.parametrize("half", [False, True])
@pytest.mark.parametrize("rep,dh", [(1, 128), (4, 64), (8, 128)])
def test_infinite_values(cuda, torch_mod, orc, rep, dh, half):
    """A value that overflowed its cache: the dims that it is in are infinite, not the product of nothing and infinity."""
    for allow in (1, 33, 1000):
        run(cuda, torch_mod, orc, 2, rep, dh, 1024, allow, half, last_v=np.inf)
        run(cuda, torch_mod, orc, 2, rep, dh, 1024, allow, half, last_v=-np.inf)
