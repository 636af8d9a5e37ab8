"""The renderer's integer marching and empty-space jumps against the CPU restatement, byte for
byte: cameras inside, outside and on the faces of the domain, rays along the axes (zero
direction components), positions that start on, fall through and cross powers of two, and
block grids whose sides are no multiples of the occupancy groups."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
CAMS = [((0.5, 0.5, -0.25), (0.5, 0.5, 0.5)), ((0.25, 0.5, 0.0), (0.25, 0.5, 1.0)), ((-0.5, 0.3, 0.4), (1.0, 0.31, 0.45)),
        ((1.5, 1.2, 1.4), (0.3, 0.2, 0.4)), ((0.9, 0.125, 0.9), (0.1, 0.12, 0.1)), ((0.03, 0.9, 0.5), (0.6, 0.0, 0.5))]


def _rgb(px):
    px = np.asarray(px, np.int64)
    return np.stack([px & 255, (px >> 8) & 255, (px >> 16) & 255], -1).astype(np.uint8)


@pytest.mark.parametrize("bsx,nb", [(8, (19, 9, 33)), (16, (17, 16, 5)), (32, (4, 9, 21)), (8, (1, 1, 1))])
@pytest.mark.parametrize("size", [(1, 1), (61, 47)])
def test_marching_matches_restatement(gpulib, port, bsx, nb, size):
    rng = np.random.Generator(np.random.PCG64(bsx + nb[2]))
    n = nb[0] * nb[1] * nb[2]
    bids = np.sort(rng.choice(n, max(1, n // 40), replace=False)).astype(np.int32)
    slot = np.full(n, -1, np.int32)
    slot[bids] = np.arange(len(bids), dtype=np.int32)
    # smooth bumps that are low on block faces, so that no ray grazes a jump of the density
    c = (np.arange(bsx) + 0.5) / bsx
    bump = np.einsum("i,j,k->ijk", *[np.sin(np.pi * c)] * 3).reshape(1, -1)
    pay = np.round(65535 * bump * rng.uniform(0.6, 1.0, (len(bids), 1))).astype(np.uint16)
    dims = [k * bsx for k in nb]
    g = gpulib.MultiresSparseGrid(*dims, bsx, 2, gpulib.U16)
    try:
        levels = np.ones(n, np.int32)
        levels[bids] = 0
        g.set_levels(levels)
        g.setRefinementMap(0.0)
        g.upload_payload(pay)
        og = port.grid(*dims, bsx, port.U16)
        for pos, look in CAMS:
            cam = {"pos": pos, "look_at": look, "sun": (0.5, 5.0, 5.0), "color": (0.8, 0.6, 0.4), "zoom": 1.3}
            got, want = g.render(0, *size, cam), _rgb(port.render(og, slot, pay, *size, cam))
            assert np.array_equal(got, want), (pos, int((got != want).any(-1).sum()))
    finally:
        g.close()
