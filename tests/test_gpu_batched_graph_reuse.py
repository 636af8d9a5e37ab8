"""The batched solve's captured iteration is not replayed once what it holds has changed: other
sweep counts or another coarsest solve give the eager path's bits, and released work vectors
give a new capture (counted in launches; no stale graph is run)."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
CH_X, CH_B, RES, BS = 1, 2, 64, 16
TOL = 1e-6


@pytest.fixture(scope="module")
def grid(gpulib):
    """Two volumes of two blocks each in opposite corners."""
    levels, vol = np.ones((4, 4, 4), np.int32), np.full((4, 4, 4), -1, np.int32)
    for v, (z, y, x) in enumerate([(0, 0, 0), (3, 3, 2)]):
        levels[z, y, x:x + 2] = 0
        vol[z, y, x:x + 2] = v
    g = gpulib.MultiresSparseGrid(RES, RES, RES, BS, 2, gpulib.F32)
    g.set_levels(levels.reshape(-1))
    g.setRefinementMap(0.0)
    for ch in (CH_X, CH_B):
        g.channel_create(ch, gpulib.F32)
    g.poisson_procedural_coefficients(31)
    g.batch_set_volumes(vol.reshape(-1), 2)
    rng = np.random.default_rng(5)
    g.upload_payload(rng.standard_normal((4, BS ** 3)).astype(np.float32), CH_B)
    yield g
    g.close()


def _solve(g, use_graph):
    g.fill(0.0, CH_X)
    before = g.launch_count()
    its, _, rel, _ = g.batch_mgpcg_solve(CH_X, CH_B, tol=TOL, max_iter=60, use_graph=use_graph)
    assert np.all(rel <= TOL)
    return its, g.payload(CH_X), g.launch_count() - before


@pytest.mark.parametrize("params", [(1, 1, 1, 0), (3, 1, 2, 0), (2, 2, 3, 40)])
def test_changed_cycle_parameters(grid, params):
    g = grid
    g.poisson_set_params()
    _solve(g, True)  # captures with the defaults
    g.poisson_set_params(*params)
    its_g, xg, _ = _solve(g, True)
    its_e, xe, _ = _solve(g, False)
    g.poisson_set_params()
    assert np.array_equal(its_g, its_e)
    assert np.array_equal(xg.view(np.uint32), xe.view(np.uint32))


def test_released_work_vectors(grid):
    g = grid
    g.poisson_set_params()
    g.poisson_release_work()
    its, x, first = _solve(g, True)  # eager first iteration, then the capture
    _, x2, replay = _solve(g, True)
    assert replay < first and np.array_equal(x, x2)
    g.poisson_release_work()
    its3, x3, again = _solve(g, True)
    assert again == first and np.array_equal(its, its3) and np.array_equal(x, x3)
