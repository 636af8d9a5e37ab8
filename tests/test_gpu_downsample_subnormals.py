"""The restriction of FP32 fields with subnormal values, bit for bit: sums that stay subnormal,
and subnormal values beside ordinary ones (weights down to 1/512 keep their low bits)."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bs,nb", [(8, 3), (16, 2), (32, 2)])
@pytest.mark.parametrize("simple", [False, True])
@pytest.mark.parametrize("share", [1.0, 0.5])
def test_subnormal_values(gpulib, port, bs, nb, simple, share):
    rng = np.random.default_rng(bs)
    g = gpulib.MultiresSparseGrid(nb * bs, nb * bs, nb * bs, bs, 2, gpulib.F32)
    try:
        g.set_levels(np.zeros(nb ** 3, np.int32))
        g.setRefinementMap(0.0)
        bids, slot = g.active_blocks().astype(np.int32), g.slots().astype(np.int32)
        v = rng.standard_normal((len(bids), bs ** 3))
        tiny = rng.random(v.shape) < share
        pay = np.where(tiny, v * 1e-39, v * 1e-37).astype(np.float32)
        assert np.all(np.abs(pay[tiny]) < np.finfo(np.float32).tiny)
        g.upload_payload(pay, 0)
        got = g.downsampleFloatChannelNew(0, simple)
    finally:
        g.close()
    og = port.grid(nb * bs, nb * bs, nb * bs, bs, port.F32)
    want = np.asarray(port.downsample(og, slot, bids, pay, simple), np.float32).reshape(got.shape)
    assert np.count_nonzero(want) > 0.9 * want.size
    assert np.array_equal(got.view(np.uint32), want.view(np.uint32))
