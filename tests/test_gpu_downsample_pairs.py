"""The restriction kernel's forms of every block edge (a thread sums two coarse cells of a
column; edge 8 leaves half a warp without cells) against the CPU restatement, bit for bit,
with signed zeros, infinities and subnormal values among the data.
"""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bs,nb", [(8, 1), (8, 5), (16, 3), (32, 2)])
@pytest.mark.parametrize("storage", ["F32", "F16", "U16"])
@pytest.mark.parametrize("simple", [False, True])
def test_column_pairs_match_restatement(gpulib, port, bs, nb, storage, simple):
    rng = np.random.default_rng(bs * 10 + nb)
    g = gpulib.MultiresSparseGrid(nb * bs, nb * bs, nb * bs, bs, 2, getattr(gpulib, storage))
    try:
        levels = (rng.random(nb ** 3) < 0.3).astype(np.int32)
        levels[0] = 0
        g.set_levels(levels)
        g.setRefinementMap(0.0)
        bids, slot = g.active_blocks().astype(np.int32), g.slots().astype(np.int32)
        n = len(bids)
        if storage == "U16":
            pay = rng.integers(0, 65536, (n, bs ** 3)).astype(np.uint16)
            host = pay
        else:
            f = rng.standard_normal((n, bs ** 3)).astype(np.float32)
            f[rng.random(f.shape) < 0.2] = -0.0
            f[rng.random(f.shape) < 0.05] *= 1e-7
            f[:, 5] = np.inf  # one sign only: no NaN, whose payload is not part of the contract
            pay = f.astype(np.float16) if storage == "F16" else f
            host = pay.view(np.uint16) if storage == "F16" else pay
        g.upload_payload(pay, 0)
        got = g.downsampleFloatChannelNew(0, simple)
    finally:
        g.close()
    og = port.grid(nb * bs, nb * bs, nb * bs, bs, getattr(port, storage))
    want = np.asarray(port.downsample(og, slot, bids, host, simple), np.float32).reshape(got.shape)
    assert np.array_equal(got.view(np.uint32), want.view(np.uint32))
