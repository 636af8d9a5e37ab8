"""The splat's list passes with four and eight particles a thread (chosen by the number of
particles) against the CPU restatement, bit for bit; counts that are no multiple of a CTA's
particles, and the last below and first above each limit."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
FOUR, EIGHT = 152 * 4 * 512 * 2, 152 * 4 * 512 * 8  # first counts with four and eight a thread


@pytest.mark.parametrize("n", [FOUR - 1, FOUR, FOUR + 77, EIGHT - 1, EIGHT, EIGHT + 333])
@pytest.mark.parametrize("storage,bsx", [("F32", 8), ("F16", 16)])
def test_many_particles(gpulib, port, n, storage, bsx):
    res, r, nb = (128 if bsx == 8 else 64), 0.5, 0.5  # 8: more blocks than the table has places
    rng = np.random.Generator(np.random.PCG64(n))
    # most on a shell, in the order of a scan over it (long lists), the rest anywhere
    u = rng.standard_normal((n, 3)).astype(np.float32)
    u /= np.linalg.norm(u, axis=1, keepdims=True)
    pts = res / 2 + (0.3 * res) * u[np.argsort(u[:, 2])]
    k = n // 8
    pts[:k] = rng.uniform(1, res - 1, (k, 3))
    pts = np.ascontiguousarray(pts, np.float32)
    g = gpulib.MultiresSparseGrid(res, res, res, bsx, 3, getattr(gpulib, storage))
    try:
        d = g.to_device(pts)
        g.mark_points(d, n, r + nb)
        g.levels_from_marks()
        g.regularizeRefinementMap()
        g.setRefinementMap(1.0)
        g.splat(d, n, r, nb)
        g.splat_finalize(r, nb)
        got = g.payload(0)
        d.free()
    finally:
        g.close()
    p = port.surface_pipeline(pts, res, bsx, storage=getattr(port, storage), n_iter=0, r_particle=r, nb_dist=nb)
    want = np.asarray(p.after_finalize).reshape(got.shape)
    bits = {2: np.uint16, 4: np.uint32}[got.dtype.itemsize]
    assert np.array_equal(got.view(bits), want.view(bits))
