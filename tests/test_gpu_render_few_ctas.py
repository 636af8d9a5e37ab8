"""The renderer's two march forms (pictures of up to 608 CTAs of 16x8 pixels step in FP64, larger
ones in integers) against the CPU restatement, byte for byte, at the last size of the one and
the first of the other, on layouts with empty space to jump and without."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
CAMS = [((0.5, 0.5, -0.25), (0.5, 0.5, 0.5)), ((0.25, 0.5, 0.0), (0.25, 0.5, 1.0)), ((1.5, 1.2, 1.4), (0.3, 0.2, 0.4))]


# CTAs: 608 = 32 x 19 and 19 x 32; 612 = 34 x 18
@pytest.mark.parametrize("size", [(512, 152), (304, 256), (544, 144), (513, 145)])
@pytest.mark.parametrize("storage", ["F32", "F16", "U16"])
@pytest.mark.parametrize("bsx,nb,share", [(8, 12, 1.0), (16, 9, 0.1), (32, 5, 0.3)])
def test_both_forms(gpulib, port, bsx, nb, share, storage, size):
    rng = np.random.Generator(np.random.PCG64(bsx))
    n = nb ** 3
    bids = np.sort(rng.choice(n, int(share * n), replace=False)).astype(np.int32)
    slot = np.full(n, -1, np.int32)
    slot[bids] = np.arange(len(bids), dtype=np.int32)
    c = (np.arange(bsx) + 0.5) / bsx
    bump = np.einsum("i,j,k->ijk", *[np.sin(np.pi * c)] * 3).reshape(1, -1) * rng.uniform(0.3, 1.0, (len(bids), 1))
    pay = {"F32": bump.astype(np.float32), "F16": bump.astype(np.float16),
           "U16": np.round(65535 * bump).astype(np.uint16)}[storage]
    g = gpulib.MultiresSparseGrid(*[nb * bsx] * 3, bsx, 2, getattr(gpulib, storage))
    try:
        levels = np.ones(n, np.int32)
        levels[bids] = 0
        g.set_levels(levels)
        g.setRefinementMap(0.0)
        g.upload_payload(pay)
        og = port.grid(*[nb * bsx] * 3, bsx, getattr(port, storage))
        host = pay.view(np.uint16) if storage == "F16" else pay
        for pos, look in CAMS:
            cam = {"pos": pos, "look_at": look, "sun": (0.5, 5.0, 5.0), "color": (0.8, 0.6, 0.4), "zoom": 1.3}
            got, px = g.render(0, *size, cam), np.asarray(port.render(og, slot, host, *size, cam), np.int64)
            want = np.stack([px & 255, (px >> 8) & 255, (px >> 16) & 255], -1).astype(np.uint8)
            assert np.array_equal(got, want), (pos, int((got != want).any(-1).sum()))
    finally:
        g.close()
