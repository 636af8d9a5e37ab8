"""Halo fills of level payloads bound at element-aligned addresses (read element by element)
give the boxes of an aligned copy, bit for bit: both forms of the fill (by rows; by planes for
edges below 8 and wide halos), the block's own level shifted, the coarser one, or both."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shift", [(1, 0), (2, 0), (3, 1), (0, 1)])
@pytest.mark.parametrize("storage", ["F32", "F16", "U16"])
@pytest.mark.parametrize("bsx,level,halo", [(8, 0, 1), (8, 0, 2), (8, 1, 1), (8, 1, 4), (16, 0, 2), (16, 0, 3),
                                            (16, 2, 1), (32, 0, 1), (32, 0, 4), (32, 1, 4)])
def test_shifted_payloads(gpulib, bsx, level, halo, storage, shift):
    G = gpulib
    rng = np.random.Generator(np.random.PCG64(bsx + halo))
    nb, st = (3, 4, 3), getattr(G, storage)
    n = nb[0] * nb[1] * nb[2]
    levels = (level + rng.integers(0, 2, n)).astype(np.int32)
    g = G.MultiresSparseGrid(*(k * bsx for k in nb), bsx, level + 2, st)
    bufs = []
    try:
        g.set_levels(levels)
        g.setRefinementMap(0.0)
        for l in (level, level + 1):
            state = np.where(rng.random(n) < 0.3, -1, -3).astype(np.int32)
            own = np.flatnonzero(levels == l)
            state[own] = np.arange(len(own))
            pay = rng.random((len(own), (bsx >> l) ** 3)).astype(np.float32)
            pay = np.round(pay * 65535).astype(np.uint16) if storage == "U16" else pay.astype(G.NP_STORAGE[st])
            g.level_grid_set(0, l, st, state, pay)
            by = shift[l - level]
            bufs += [g.to_device(state), g.to_device(np.concatenate([np.zeros(by, pay.dtype), pay.ravel()]))]
            g.level_grid_bind(1, l, st, bufs[-2].ptr, bufs[-1].ptr + by * pay.itemsize)
        bids = np.flatnonzero(levels == level).astype(np.int32)
        for opt in (0, G.BC_NEUMANN, G.BC_COARSE_LEVEL):
            want, skip = g.fill_halo_blocks(0, level, bids, halo, opt)
            got, skip1 = g.fill_halo_blocks(1, level, bids, halo, opt)
            assert skip == skip1 == 0
            assert np.array_equal(got.view(np.uint32), want.view(np.uint32))
    finally:
        for b in bufs:
            b.free()
        g.close()
