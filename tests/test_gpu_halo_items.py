"""The halo fill's thread-per-item form: a coarser level bound at an element-aligned address
(which it leaves to the other form; the block's own level is read in 16-byte rows by both and
must be aligned so) gives the boxes of an aligned copy, bit for bit, for every option."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shift", [(0, 0), (0, 1), (0, 3)])
@pytest.mark.parametrize("storage", ["F32", "F16", "U16"])
@pytest.mark.parametrize("bsx,halo", [(8, 1), (16, 3), (32, 2), (32, 3)])
def test_element_aligned_levels(gpulib, bsx, halo, storage, shift):
    G = gpulib
    rng = np.random.Generator(np.random.PCG64(bsx + halo))
    nb, st = (3, 4, 3), getattr(G, storage)
    n = nb[0] * nb[1] * nb[2]
    levels = rng.integers(0, 2, n).astype(np.int32)
    g = G.MultiresSparseGrid(*(k * bsx for k in nb), bsx, 2, st)
    bufs = []
    try:
        g.set_levels(levels)
        g.setRefinementMap(0.0)
        for l in range(2):
            state = np.where(levels == l, 0, np.where(rng.random(n) < 0.3, -1, -3)).astype(np.int32)
            own = np.flatnonzero(levels == l)
            state[own] = np.arange(len(own))
            pay = rng.random((len(own), (bsx >> l) ** 3)).astype(np.float32)
            pay = np.round(pay * 65535).astype(np.uint16) if storage == "U16" else pay.astype(G.NP_STORAGE[st])
            g.level_grid_set(0, l, st, state, pay)
            off = np.concatenate([np.zeros(shift[l], pay.dtype), pay.ravel()])
            bufs += [g.to_device(state), g.to_device(off)]
            g.level_grid_bind(1, l, st, bufs[-2].ptr, bufs[-1].ptr + shift[l] * pay.itemsize)
        bids = np.flatnonzero(levels == 0).astype(np.int32)
        for opt in (0, G.BC_NEUMANN, G.BC_COARSE_LEVEL):
            want, skip = g.fill_halo_blocks(0, 0, bids, halo, opt)
            got, skip1 = g.fill_halo_blocks(1, 0, bids, halo, opt)
            assert skip == skip1 == 0
            assert np.array_equal(got.view(np.uint32), want.view(np.uint32))
    finally:
        for b in bufs:
            b.free()
        g.close()
