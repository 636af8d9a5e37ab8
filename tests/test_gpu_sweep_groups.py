"""The sweep kernel's z-group forms (one, two or four groups of planes per block, chosen by
the number of blocks in a colour pass) against the CPU restatement, bit for bit.

Layouts lie on both sides of each limit of the rule; a few blocks hold no payload, so every
group meets neighbours of each kind (value block, empty block, domain boundary).  Values
include runs of equal ones (zero gradients) and the range's ends.
"""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
OPT8 = 1 << 29
MCF8, JAC8, LAPL8 = -(4 + OPT8), -(17 + OPT8), -(1 + OPT8)


def _field(rng, n, vox, storage):
    f = rng.random((n, vox), np.float32)
    f[:, : vox // 4] = np.round(f[:, : vox // 4] * 3) / 3
    if storage == "U16":
        return np.round(f * 65535).astype(np.uint16)
    return f.astype(np.float16) if storage == "F16" else f


# blocks a pass: 8 and 152 (four groups on 16^3 blocks, two on 32^3), 343 (two), 729 (one)
CASES = [(16, 4, "F32", MCF8), (16, 4, "U16", MCF8), (16, 4, "F16", JAC8), (16, 4, "U16", LAPL8),
         (16, 14, "F32", MCF8), (16, 14, "U16", MCF8), (16, 18, "F32", MCF8), (16, 18, "F16", MCF8),
         (16, 14, "F32", JAC8), (32, 4, "F16", MCF8), (32, 4, "F16", JAC8), (32, 4, "F32", MCF8),
         (32, 11, "U16", MCF8), (32, 11, "F32", MCF8)]


@pytest.mark.parametrize("bsx,nb,storage,lapl", CASES)
def test_group_forms_match_restatement(gpulib, port, bsx, nb, storage, lapl):
    rng = np.random.Generator(np.random.PCG64(bsx * 1000 + nb))
    levels = (rng.random(nb ** 3) < 0.04).astype(np.int32)
    g = gpulib.MultiresSparseGrid(nb * bsx, nb * bsx, nb * bsx, bsx, 2, getattr(gpulib, storage))
    try:
        g.set_levels(levels)
        g.setRefinementMap(0.0)
        bids, slot = g.active_blocks(), g.slots()
        f = _field(rng, len(bids), bsx ** 3, storage)
        g.upload_payload(f)
        g.applyChannelPdeFast(0, laplTyp=lapl, doConstrZeroOne=1, numIter=2, timeStep=0.1)
        got = g.payload(0)
    finally:
        g.close()
    og = port.grid(nb * bsx, nb * bsx, nb * bsx, bsx, getattr(port, storage))
    want = port.pde(og, slot, bids, f.copy(), lapl, 1, 2, 0.1)
    bits = {2: np.uint16, 4: np.uint32}[got.dtype.itemsize]
    assert np.array_equal(got.view(bits), np.asarray(want).reshape(got.shape).view(bits))
