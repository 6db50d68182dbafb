"""The GEMM on serialized blocks, at the edges of its dispatch: row tiles of 128, groups of 256 weights, token
tiles, tiles shared by a cluster along K, rows on and off the 16-byte grid."""
from __future__ import annotations

import ctypes as C
import os
import subprocess
import sys

import numpy as np
import pytest

from tensormark_b200 import lib, synth
from tests.gpu_util import dev_f32, ptr, stream_ptr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dt,m,n,k,shift", [
    (synth.Q4_0, 1, 1, 32, 0), (synth.Q4_0, 2, 127, 256, 0), (synth.Q4_0, 17, 129, 288, 0), (synth.Q4_0, 16, 4096, 1024, 0),
    (synth.Q4_0, 33, 257, 2080, 0), (synth.Q4_0, 65, 300, 4096, 0), (synth.Q4_0, 129, 1000, 512, 0), (synth.Q4_0, 256, 256, 8192, 0),
    (synth.Q4_0, 20, 256, 2048, 2), (synth.Q4_0, 5, 9500, 2048, 0), (synth.Q4_0, 90, 19000, 512, 0),
    (synth.GGUF_Q4_0, 12, 200, 4128, 0), (synth.GGUF_Q4_0, 70, 256, 512, 6),
    (synth.Q4_1, 9, 130, 544, 0), (synth.Q4_1, 100, 384, 2048, 0), (synth.Q4_1, 31, 384, 2048, 4),
    (synth.Q8_0, 3, 200, 2112, 0), (synth.Q8_0, 48, 3000, 1024, 0), (synth.Q8_0, 8, 96, 14336, 1),
    (synth.Q6_K, 20, 5119, 256, 0), (synth.Q6_K, 77, 300, 2816, 0), (synth.Q6_K, 4, 128, 14336, 3),
    (synth.Q5_K, 6, 250, 14336, 0), (synth.Q5_K, 128, 512, 768, 0), (synth.Q4_K, 3, 129, 256, 0), (synth.Q4_K, 200, 640, 4096, 0),
    (synth.Q5_K, 20, 250, 512, 2), (synth.Q4_K, 20, 250, 512, 1), (synth.Q4_0, 512, 300, 1024, 0), (synth.Q6_K, 511, 257, 512, 0),
    # past the last token count it takes: the fp16 copy, eight weights per thread
    (synth.Q4_0, 513, 130, 544, 0), (synth.GGUF_Q4_0, 513, 130, 544, 0), (synth.Q4_1, 513, 130, 544, 0), (synth.Q8_0, 513, 130, 544, 0),
    (synth.Q4_K, 513, 130, 768, 0), (synth.Q5_K, 513, 130, 768, 0), (synth.Q6_K, 513, 130, 768, 0), (synth.Q8_0, 513, 130, 544, 1),
])
def test_edges(cuda, torch_mod, orc, dt, m, n, k, shift):
    torch = torch_mod
    W = synth.make_weights(dt, n, k, seed=14)
    A = synth.make_activations((m, k), seed=15)
    flat = np.ascontiguousarray(W, dtype=np.uint8).reshape(-1)
    Wd = torch.zeros(flat.size + 64, dtype=torch.uint8, device="cuda")
    Wd[shift:shift + flat.size] = torch.from_numpy(flat).cuda()
    Ad = dev_f32(torch, A)
    Cd = torch.full((m + 1, n), float("nan"), dtype=torch.float32, device="cuda")
    need = cuda.tm_cuda_sgemm_q_workspace(m, n, k, dt)
    ws = torch.empty(need + 256, dtype=torch.uint8, device="cuda")
    base = C.c_void_p((ws.data_ptr() + 255) // 256 * 256)
    for _ in range(2):
        lib.check(cuda.tm_cuda_sgemm_q_dev(ptr(Ad), C.c_void_p(Wd.data_ptr() + shift), ptr(Cd), m, n, k, dt, base, need, stream_ptr(torch)),
                  "tm_cuda_sgemm_q_dev")
    torch.cuda.synchronize()
    got = Cd.cpu().numpy()
    assert np.isnan(got[m]).all()                          # nothing behind the result
    ref = orc.gemm(dt, W, A, m, n, k, threads=4)
    absum = np.abs(A) @ np.abs(orc.dequant(dt, W, n * k).reshape(n, k)).T
    err = np.abs(got[:m] - ref)
    assert np.all(err <= 1e-3 * absum), float((err / absum).max())


@pytest.mark.parametrize("dt,m,n,k", [(synth.Q4_0, 512, 32, 288), (synth.Q8_0, 400, 16, 96), (synth.Q4_0, 512, 300, 1024), (synth.Q4_0, 300, 130, 64)])
def test_scratch_size_does_not_choose_the_kernel(cuda, torch_mod, orc, dt, m, n, k):
    """A call's bits come from its operands: also where the fp16 tokens, K rounded up to 64, need more than the scratch that
    the call asks for."""
    torch = torch_mod
    W, A = synth.make_weights(dt, n, k, seed=24), synth.make_activations((m, k), seed=25)
    Wd = torch.from_numpy(np.ascontiguousarray(np.concatenate([W.reshape(-1), np.zeros(32, np.uint8)]))).cuda()
    Ad = dev_f32(torch, A)
    need = cuda.tm_cuda_sgemm_q_workspace(m, n, k, dt)
    ws = torch.empty(2 * need + (1 << 20), dtype=torch.uint8, device="cuda")
    base = C.c_void_p((ws.data_ptr() + 255) // 256 * 256)
    got = []
    for size in (need, 2 * need + (1 << 19)):
        Cd = torch.empty((m, n), dtype=torch.float32, device="cuda")
        lib.check(cuda.tm_cuda_sgemm_q_dev(ptr(Ad), ptr(Wd), ptr(Cd), m, n, k, dt, base, size, stream_ptr(torch)), "tm_cuda_sgemm_q_dev")
        torch.cuda.synchronize()
        got.append(Cd.cpu().numpy())
    assert np.array_equal(got[0], got[1])
    absum = np.abs(A) @ np.abs(orc.dequant(dt, W, n * k).reshape(n, k)).T
    assert np.all(np.abs(got[0] - orc.gemm(dt, W, A, m, n, k, threads=4)) <= 1e-3 * absum)


@pytest.mark.parametrize("env,launches", [({}, 1), ({"TM_GEMM_FUSED": "0", "TM_GEMM_BN": ""}, 1), ({"TM_GEMM_FUSED": "1"}, 2), ({"TM_GEMM_PAIR": "0"}, 2)])
def test_knobs(env, launches):
    """A few tokens are one launch, and a knob that is off leaves it at that."""
    code = ("import numpy as np, torch\n"
            "from tensormark_b200 import lib, synth\n"
            "L = lib.load()\n"
            "lib.check(L.tm_cuda_init(-1), 'tm_cuda_init')\n"
            "W, A, C = synth.make_weights(synth.Q4_0, 256, 512, seed=1), synth.make_activations((17, 512), seed=2), np.empty((17, 256), np.float32)\n"
            "before = L.tm_cuda_launch_count()\n"
            "lib.check(L.tm_cuda_sgemm_q4(A.ctypes.data, W.ctypes.data, C.ctypes.data, 17, 256, 512), 'tm_cuda_sgemm_q4')\n"
            "print(L.tm_cuda_launch_count() - before)\n")
    clean = {k: v for k, v in os.environ.items() if not k.startswith("TM_GEMM")}
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", code], cwd=root, env={**clean, **env}, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr
    assert int(r.stdout) == launches
