"""The warm start on 8^3 blocks, whose level-1 blocks of edge 4 take the forward and backward
convolutions that gather per tap: output, loss and gradients against the CPU restatement, with
the bounds of the larger blocks' test."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import rel_l2
from msbg_gb300 import workloads as W
from test_gpu_warmnet import WN, _level1_diag, _rand

pytestmark = pytest.mark.gpu
CH_X, CH_B, CH_XS = 1, 2, 3


@pytest.mark.parametrize("loss", ["coarse", "residual"])
def test_edge_4_matches_restatement(gpulib, port, loss):
    G, res, bs = gpulib, 64, 8
    pts = W.sphere_cloud(res, 4, 2000, seed=W.workload_seed(4, 1))
    g = G.MultiresSparseGrid(res, res, res, bs, 3, G.F32)
    try:
        d = g.to_device(pts)
        g.mark_points(d, len(pts), 3.0)
        g.levels_from_marks()
        g.regularizeRefinementMap()
        g.setRefinementMap(0.0)
        d.free()
        for ch in (CH_X, CH_B, CH_XS):
            g.channel_create(ch, G.F32)
        g.poisson_procedural_coefficients(4242)
        prob = port.PoissonProblem(g.active_blocks().astype(np.int64), (g.nbx, g.nby, g.nbz), bs, seed=4242)
        rng = np.random.default_rng(11)
        b = _rand(prob, rng).astype(np.float32)
        xs = (_rand(prob, rng) * 0.2).astype(np.float32)
        g.upload_payload(prob.payload(b), CH_B)
        g.upload_payload(prob.payload(xs), CH_XS)
        net = WN.WarmNet.init(123)
        net.c = [np.linspace(-0.05, 0.05, c).astype(np.float32) for c in WN.CH[1:]]
        g.warmnet_set(net.W, net.c)
        g.warmnet_set_loss(loss)
        L, gW, gc, x0 = WN.loss_and_grads(net, b.astype(np.float64), xs.astype(np.float64),
                                          (prob.act > 0).astype(np.float64), prob.apply, _level1_diag(prob), loss=loss,
                                          act_bf16=True)
        g.warmnet_predict(CH_B, CH_X)
        assert rel_l2(prob.dense(g.payload(CH_X)), x0) < 2e-4
        got, gW_gpu, gc_gpu = g.warmnet_loss_grad(CH_B, CH_XS)
        assert abs(got - L) <= 2e-4 * L
        for l in range(4):
            assert rel_l2(gW_gpu[l], gW[l]) < 2e-3, l
            assert rel_l2(gc_gpu[l], gc[l]) < 2e-3, l
    finally:
        g.close()
