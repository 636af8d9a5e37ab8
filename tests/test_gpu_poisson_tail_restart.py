"""The small levels' grid barrier carries nothing from launch to launch: after a bounded wait
gave up, which can leave any count behind, V-cycles and solves (FP32 and mixed, single and
batched through the captured graph) give the bits that they gave before."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
CH_X, CH_B, BS, NB = 1, 2, 16, (6, 6, 8)


def test_counts_left_behind_change_nothing(gpulib):
    G = gpulib
    n = NB[0] * NB[1] * NB[2]
    g = G.MultiresSparseGrid(*(k * BS for k in NB), BS, 2, G.F32)
    try:
        g.set_levels(np.zeros(n, np.int32))
        g.setRefinementMap(0.0)
        for ch in (CH_X, CH_B):
            g.channel_create(ch, G.F32)
        g.poisson_procedural_coefficients(8)
        g.batch_set_volumes(np.zeros(n, np.int32), 1)
        b = np.random.default_rng(2).standard_normal((n, BS ** 3)).astype(np.float32)
        g.upload_payload(b, CH_B)
        assert 8192 < g.mg_info()[2] <= 1 << 20  # the first level of the tail: many CTAs

        def start():
            g.fill(0.0, CH_X)

        calls = [lambda: g.vcycle(CH_X, CH_B),
                 lambda: (start(), g.mgpcg_solve(CH_X, CH_B, tol=1e-6, max_iter=50)),
                 lambda: (start(), g.mgpcg_solve_mixed(CH_X, CH_B, tol=1e-6)),
                 lambda: (start(), g.batch_mgpcg_solve(CH_X, CH_B, tol=1e-6, max_iter=50))]
        for call in calls:
            call()
            want = g.payload(CH_X)
            for _ in range(2):
                with pytest.raises(G.MsbgGpuError) as e:
                    g.diag_wait_timeout(100)
                assert e.value.code == G.ERR_TIMEOUT
                call()
                assert np.array_equal(g.payload(CH_X).view(np.uint32), want.view(np.uint32))
    finally:
        g.close()
