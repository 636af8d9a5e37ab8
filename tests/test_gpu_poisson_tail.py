"""The small levels of the V-cycle in one launch (poisson_tail.cu) against the FP64
restatement, on layouts whose levels fall on both sides of its limits: one block (every level
in one CTA), levels just above and below what one CTA holds (8192 cells), isolated blocks
whose aggregated levels hardly shrink, and other sweep counts.  Tolerance as for the V-cycle
on the dense-ish layouts: FP32 rounding through a cycle, rel-L2 1e-5."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu
CH_X, CH_B = 1, 2


# block edge, block grid, blocks: cells of the bs-4 level are 64 times the blocks
@pytest.mark.parametrize("bs,nb,n", [(8, (3, 3, 3), 1), (8, (8, 6, 5), 127), (8, (8, 6, 5), 130), (16, (9, 7, 6), 300),
                                     (8, (24, 23, 22), 900), (8, (40, 2, 2), 160)])
@pytest.mark.parametrize("params", [(2, 2, 3), (1, 1, 1)])
def test_vcycle_of_small_levels(gpulib, port, bs, nb, n, params):
    rng = np.random.Generator(np.random.PCG64(n))
    total = nb[0] * nb[1] * nb[2]
    bids = np.sort(rng.choice(total, n, replace=False)).astype(np.int64)
    levels = np.ones(total, np.int32)
    levels[bids] = 0
    g = gpulib.MultiresSparseGrid(*(k * bs for k in nb), bs, 2, gpulib.F32)
    try:
        g.set_levels(levels)
        g.setRefinementMap(0.0)
        for ch in (CH_X, CH_B):
            g.channel_create(ch, gpulib.F32)
        g.poisson_procedural_coefficients(99)
        g.poisson_set_params(*params, 0)
        prob = port.PoissonProblem(bids, nb, bs, seed=99, pre=params[0], post=params[1], tile_iters=params[2])
        b = np.where(prob.act > 0, rng.standard_normal(prob.act.shape), 0.0).astype(np.float32)
        g.upload_payload(prob.payload(b), CH_B)
        want, nlev = prob.vcycle(b)
        assert len(g.mg_info()) == nlev
        for _ in range(2):  # the barrier's counters are back at zero after a cycle
            g.vcycle(CH_X, CH_B)
            assert rel_l2(prob.dense(g.payload(CH_X)), want) < 1e-5
    finally:
        g.close()
