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


# blocks a pass: 8 (four groups on 16^3 blocks, two on 32^3), 166 on 32^3 (FP32 two, else one), 343 (two), 729 (one)
CASES = [(16, 4, "F32", MCF8), (16, 4, "U16", MCF8), (16, 4, "F16", JAC8), (16, 4, "U16", LAPL8),
         (16, 14, "F32", MCF8), (16, 14, "U16", MCF8), (16, 18, "F32", MCF8), (16, 18, "F16", MCF8),
         (16, 14, "F32", JAC8), (16, 18, "U16", JAC8), (32, 4, "F16", MCF8), (32, 4, "F16", JAC8), (32, 4, "F32", MCF8),
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


# The fast forms re-associate: within the bound that the surface tests hold them to (FP32).  An
# FP32 difference of some 2^-21 turns the FP16 rounding of at most one value in 2^9, by 2^-11:
# 2^-11 * 2^-4.5 = 2.2e-5 of the field's norm a pass, 1e-4 over two iterations of eight colours.
@pytest.mark.parametrize("nb", [4, 14, 18])
@pytest.mark.parametrize("storage,tol", [("F32", 1e-5), ("F16", 1e-4)])
@pytest.mark.parametrize("lapl,clamp", [(MCF8, 1), (MCF8, 0), (JAC8, 1), (JAC8, 0)])
def test_fast_group_forms_within_bound(gpulib, port, nb, storage, tol, lapl, clamp):
    bsx = 16
    rng = np.random.Generator(np.random.PCG64(nb * 10 + clamp))
    levels = (rng.random(nb ** 3) < 0.04).astype(np.int32)
    g = gpulib.MultiresSparseGrid(nb * bsx, nb * bsx, nb * bsx, bsx, 2, getattr(gpulib, storage))
    try:
        g.set_levels(levels)
        g.setRefinementMap(0.0)
        bids, slot = g.active_blocks(), g.slots()
        f = _field(rng, len(bids), bsx ** 3, storage)
        g.upload_payload(f)
        g.applyChannelPdeFast(0, laplTyp=lapl, doConstrZeroOne=clamp, numIter=2, timeStep=0.1,
                              variant=gpulib.SWEEP_FAST)
        got = g.payload(0).astype(np.float64)
    finally:
        g.close()
    og = port.grid(nb * bsx, nb * bsx, nb * bsx, bsx, getattr(port, storage))
    want = np.asarray(port.pde(og, slot, bids, f.copy(), lapl, clamp, 2, 0.1)).reshape(got.shape).astype(np.float64)
    assert np.linalg.norm(got - want) <= tol * np.linalg.norm(want)
