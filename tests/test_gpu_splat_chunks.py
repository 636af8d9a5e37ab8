"""The splat's chunked lists and hashed counters against the CPU restatement, bit for bit:
one block's list at, just below and above the chunk length (32 bs) and many chunks long, all
particles in one spot, particles on block corners (eight lists), enough particles per CTA
and distinct blocks to fill its hash table, and FP32 channels that keep their values."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("storage", ["F32", "F16"])
@pytest.mark.parametrize("bsx", [8, 16, 32])
@pytest.mark.parametrize("count", ["chunk-1", "chunk", "chunk+1", "many", "corners", "spread"])
def test_splat_lists_match_restatement(gpulib, port, bsx, count, storage):
    rng = np.random.Generator(np.random.PCG64(bsx))
    res, chunk = 8 * bsx, 32 * bsx
    r, nb = (1.5, 1.0) if bsx == 8 else (2.0, 2.0)
    if count == "corners":
        pts = bsx * rng.integers(1, 8, (3000, 3)) + rng.uniform(-0.3, 0.3, (3000, 3))
    elif count == "spread":
        res = 32 * bsx
        pts = rng.uniform(1, res - 1, (40000 if bsx == 8 else 9000, 3))
    else:
        n = {"chunk-1": chunk - 1, "chunk": chunk, "chunk+1": chunk + 1, "many": 9 * chunk + 5}[count]
        pts = 3.5 * bsx + rng.uniform(-0.1, 0.1, (n, 3)) * bsx
    pts = np.ascontiguousarray(pts, np.float32)
    g = gpulib.MultiresSparseGrid(res, res, res, bsx, 3, getattr(gpulib, storage))
    try:
        d = g.to_device(pts)
        g.mark_points(d, len(pts), r + nb)
        g.levels_from_marks()
        g.regularizeRefinementMap()
        g.setRefinementMap(1.0)
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
