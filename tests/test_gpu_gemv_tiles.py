"""The streaming GEMV at the edges of its tiling: tiles of 16 rows, groups of 256 weights, chunks of groups, rows on and
off the 16-byte grid. Same checker and bars as the other GEMV tests."""
from __future__ import annotations

import numpy as np
import pytest

from tensormark_b200 import synth
from tests.bounds import activation_rounding_bound
from tests.gpu_util import dev_bytes, dev_f32, gemv_dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dt,n,k", [
    (synth.Q4_0, 1, 256), (synth.Q8_0, 17, 768), (synth.Q4_1, 16 * 148 + 1, 512),        # many teams; one row over a tile
    (synth.Q4_0, 33, 4096), (synth.Q4_0, 33, 4352), (synth.Q8_0, 31, 10240),             # one chunk, one group over, several
    (synth.Q6_K, 2400, 2048), (synth.Q6_K, 40, 18432), (synth.Q5_K, 15, 14592), (synth.Q4_K, 47, 8192),
    (synth.Q4_0, 300, 32), (synth.Q4_0, 5000, 2080), (synth.Q8_0, 77, 4128), (synth.Q4_1, 50, 14368),   # rows off the grid
    (synth.GGUF_Q4_0, 19, 352), (synth.Q6_K, 149, 2816), (synth.Q6_K, 3, 14592),
])
def test_tile_edges(cuda, torch_mod, orc, dt, n, k):
    W = synth.make_weights(dt, n, k, seed=80)
    x = synth.make_activations(k, seed=81)
    y = gemv_dev(cuda, torch_mod, dt, dev_bytes(torch_mod, W), dev_f32(torch_mod, x), n, k)
    y64, yabs = orc.gemv_f64(dt, W, x, n, k)
    err = np.abs(y - y64)
    assert np.all(err <= activation_rounding_bound(orc, dt, W, x, n, k) + 2e-6 * yabs), float((err / yabs).max())
    if W.shape[1] % 16:                        # there x is held as closely as fp32 does
        assert np.all(err <= 2e-6 * yabs), float((err / yabs).max())


@pytest.mark.parametrize("n,k", [(33, 33024), (5, 49152)])
def test_longer_than_the_planes_serve(cuda, torch_mod, orc, n, k):
    """Beyond 32768 activations x is multiplied in fp32: a large one under a weight of zero costs its neighbours nothing."""
    W = synth.make_weights(synth.Q4_0, n, k, seed=82)
    first = W.reshape(n, k // 32, 18)[:, :, 2]
    first[:] = (first & 0xF0) | 8              # the block's first weight is zero
    x = synth.make_activations(k, seed=83)
    x[::32] = 1000.0
    y = gemv_dev(cuda, torch_mod, synth.Q4_0, dev_bytes(torch_mod, W), dev_f32(torch_mod, x), n, k)
    y64, yabs = orc.gemv_f64(synth.Q4_0, W, x, n, k)
    err = np.abs(y - y64)
    assert np.all(err <= 2e-6 * yabs), float((err / yabs).max())
