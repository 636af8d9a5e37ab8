"""The small levels of the V-cycle: layouts whose first pointwise level is just within and just
above what the one launch takes (2^20 cells), against the FP64 restatement with the V-cycle
tests' bound, and the FP16-storage form, which the mixed solve runs, against the same cycle in
separate launches."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu
CH_X, CH_B = 1, 2


def _grid(gpulib, bs, nb, n, seed):
    rng = np.random.Generator(np.random.PCG64(seed))
    total = nb[0] * nb[1] * nb[2]
    bids = np.sort(rng.choice(total, n, replace=False)).astype(np.int64)
    levels = np.ones(total, np.int32)
    levels[bids] = 0
    g = gpulib.MultiresSparseGrid(*(k * bs for k in nb), bs, 2, gpulib.F32)
    g.set_levels(levels)
    g.setRefinementMap(0.0)
    for ch in (CH_X, CH_B):
        g.channel_create(ch, gpulib.F32)
    g.poisson_procedural_coefficients(99)
    return g, bids, rng


@pytest.mark.parametrize("n", [16384, 16385])
def test_vcycle_at_the_cell_limit(gpulib, port, n):
    bs, nb = 8, (26, 26, 25)
    g, bids, rng = _grid(gpulib, bs, nb, n, 5)
    try:
        g.poisson_set_params(1, 1, 1, 0)
        prob = port.PoissonProblem(bids, nb, bs, seed=99, pre=1, post=1, tile_iters=1)
        b = np.where(prob.act > 0, rng.standard_normal(prob.act.shape), 0.0).astype(np.float32)
        g.upload_payload(prob.payload(b), CH_B)
        want, nlev = prob.vcycle(b)
        assert len(g.mg_info()) == nlev and g.mg_info()[1] == 64 * n
        g.vcycle(CH_X, CH_B)
        assert rel_l2(prob.dense(g.payload(CH_X)), want) < 1e-5
    finally:
        g.close()


# One outer step of one inner iteration: x = alpha M b with the FP16 cycle M.  The two forms hold
# x and b of every level in FP16 (unit roundoff 2^-11) and differ in the roundings of residuals
# and in the coarsest solve; errors of the levels add, some 20 of these roundings in all: 1e-2.
@pytest.mark.parametrize("bs,nb,n", [(8, (3, 3, 3), 5), (8, (8, 6, 5), 127), (8, (8, 6, 5), 240), (16, (9, 7, 6), 300)])
def test_fp16_form_matches_separate_launches(gpulib, bs, nb, n):
    g, bids, rng = _grid(gpulib, bs, nb, n, n)
    try:
        g.upload_payload(rng.standard_normal((n, bs ** 3)).astype(np.float32), CH_B)
        x, launches = [], []
        for coarsest in (0, 400):  # 0: exact, all small levels in one launch; else one launch a half sweep
            g.poisson_set_params(2, 2, 3, coarsest)
            g.fill(0.0, CH_X)
            before = g.launch_count()
            g.mgpcg_solve_mixed(CH_X, CH_B, tol=1e-12, max_outer=1, inner_tol=1e-3, max_inner=1)
            launches.append(g.launch_count() - before)
            v = g.payload(CH_X).astype(np.float64)
            x.append(v / np.linalg.norm(v))
        assert launches[0] < launches[1] - 40
        assert rel_l2(x[0], x[1]) < 1e-2
    finally:
        g.close()
