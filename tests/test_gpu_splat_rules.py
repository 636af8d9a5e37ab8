"""The splat's launch rules against the CPU restatement, bit for bit: whole warps per particle
(wide boxes; fewer particles than a block has warps), and one block's list on layouts whose
blocks fill the chip, just below, at and above the count from which lists are split, and many
chunks long."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _check(gpulib, port, pts, res, bsx, storage, r, nb):
    pts = np.ascontiguousarray(pts, np.float32)
    g = gpulib.MultiresSparseGrid(res, res, res, bsx, 3, getattr(gpulib, storage))
    try:
        d = g.to_device(pts)
        g.mark_points(d, len(pts), r + nb)
        g.levels_from_marks()
        g.regularizeRefinementMap()
        g.setRefinementMap(1.0)
        n_act = int(g.info().nActive)
        g.splat(d, len(pts), r, nb)
        g.splat_finalize(r, nb)
        got = g.payload(0)
        d.free()
    finally:
        g.close()
    p = port.surface_pipeline(pts, res, bsx, storage=getattr(port, storage), n_iter=0, r_particle=r, nb_dist=nb)
    want = np.asarray(p.after_finalize).reshape(got.shape)
    bits = {2: np.uint16, 4: np.uint32}[got.dtype.itemsize]
    assert np.array_equal(got.view(bits), want.view(bits))
    return n_act


# radius + band: 5 is the last box of half warps (11 rows of 11), 5.5 the first of whole ones
@pytest.mark.parametrize("storage", ["F32", "F16", "U16"])
@pytest.mark.parametrize("bsx,r,nb", [(16, 3.0, 2.0), (16, 3.5, 2.0), (16, 5.0, 2.5), (32, 6.0, 4.0), (32, 9.0, 6.5)])
@pytest.mark.parametrize("n", [9, 6000])
def test_wide_boxes(gpulib, port, bsx, r, nb, storage, n):
    rng = np.random.Generator(np.random.PCG64(n))
    res = 6 * bsx
    u = rng.standard_normal((n, 3))
    _check(gpulib, port, res / 2 + 0.2 * res * u / np.linalg.norm(u, axis=1, keepdims=True), res, bsx, storage, r, nb)


@pytest.mark.parametrize("storage", ["F32", "F16"])
@pytest.mark.parametrize("bsx,nblk", [(8, 10), (16, 8), (32, 5)])
@pytest.mark.parametrize("count", [-1, 0, 1, 12345])
def test_long_lists_on_wide_layouts(gpulib, port, bsx, nblk, storage, count):
    rng = np.random.Generator(np.random.PCG64(bsx))
    res = nblk * bsx
    c = (np.arange(nblk) + 0.5) * bsx
    every = np.stack(np.meshgrid(c, c, c), -1).reshape(-1, 3)  # one particle in every block
    n = 4 * 32 * bsx + count - nblk ** 3  # particles in all: those in every block are part of the count
    spot = 3.5 * bsx + rng.uniform(-0.1, 0.1, (n, 3)) * bsx
    n_act = _check(gpulib, port, np.concatenate([spot, every]), res, bsx, storage, 1.5, 1.0)
    assert n_act == nblk ** 3 and n_act * (2 if bsx == 32 else 1) > 152 * 1536 // (16 * bsx) // 2
