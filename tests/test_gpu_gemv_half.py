"""The 16-bit GEMV over the ways it shares a row out: eight lanes, one to eight warps, rows that leave lanes idle, more rows than
one wave of CTAs."""
from __future__ import annotations

import numpy as np
import pytest

from tensormark_b200 import synth
from tests.gpu_util import dev_f32, gemv_dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dt", [synth.F16, synth.BF16])
@pytest.mark.parametrize("n,k", [
    (1, 8), (3, 256), (1200, 8), (4737, 1024), (4736, 1024), (20000, 520), (40, 1032), (105, 3584), (300, 2048), (900, 2040), (75, 16384), (1000, 14336),
    (5000, 4104), (6, 50000), (12, 100), (9, 4097),
])
def test_row_shares(cuda, torch_mod, dt, n, k):
    torch = torch_mod
    g = torch.Generator(device="cuda").manual_seed(n)
    w = (torch.randn(n, k, generator=g, device="cuda") * 0.05).to(torch.float16 if dt == synth.F16 else torch.bfloat16)
    x = np.random.default_rng(k).standard_normal(k).astype(np.float32)
    y = gemv_dev(cuda, torch, dt, w, dev_f32(torch, x), n, k)
    wd = w.double().cpu().numpy()
    assert np.all(np.abs(y - wd @ x) <= 2e-6 * (np.abs(wd) @ np.abs(x)))


@pytest.mark.parametrize("dt", [synth.F16, synth.BF16])
def test_weights_from_the_kernel_before(cuda, torch_mod, dt):
    """W may be the output of the launch right before, as x may: merged weights, for instance."""
    torch = torch_mod
    n, k, r = 1500, 2048, 64
    g = torch.Generator(device="cuda").manual_seed(5)
    t = torch.float16 if dt == synth.F16 else torch.bfloat16
    w, x = torch.empty(n, k, dtype=t, device="cuda"), torch.randn(k, generator=g, device="cuda")
    for _ in range(20):
        a, b = (torch.randn(*s, generator=g, device="cuda").to(t) for s in ((n, r), (r, k)))
        w.zero_()
        torch.cuda.synchronize()
        torch.matmul(a, b, out=w)
        y = gemv_dev(cuda, torch, dt, w, x, n, k)
        assert np.array_equal(y, gemv_dev(cuda, torch, dt, w, x, n, k))
