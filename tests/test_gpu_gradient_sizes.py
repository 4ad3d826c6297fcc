"""Proposal gradients at the sizes where the training kernels' tiles end: one,
two and three chunks of 64 clusters (the per-chunk pipeline with no, one and
several refills of its weight tiles) and row counts around the 128-row tile,
against the oracle's double-precision gradient with bf16 rounding at the points
where the product rounds.

Tolerance: the sums differ only in the order of FP32 additions (below 1e-5
relative here) and where an FP32 and a double sum straddle a bf16 rounding
boundary: one bf16 step, 2^-8 relative, of one hidden value or logit gradient.
A single row has 64 hidden values a layer, and a block's relative L2 error is
at most that of all of them off by one step in each of three layers,
3 * 2^-8 < 2e-2.
"""
from __future__ import annotations

import numpy as np
import pytest

import oracle_binding as ob
from helpers import mlp_params

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def small(restir_lib):
    from restir_gb300 import scenes
    s = scenes.config2(width=64, height=48, n_tris=2000, n_lights=1024, frames=1)
    return s, scenes.trace_gbuffer_host(s, 0)


@pytest.mark.parametrize("clusters", [64, 128, 192])
@pytest.mark.parametrize("n", [1, 127, 128, 129, 257])
def test_gradients_at_tile_edges(ctx, small, cuda, clusters, n):
    from restir_gb300.passes import DeviceGBuffer
    from restir_gb300._lib import RestirError
    s, g = small
    cluster_of = (np.arange(len(s.point_lights)) % clusters).astype(np.int32)
    ctx.upload_scene(s)
    ctx.create_proposal(cluster_of, clusters, mix=0.9, batch=256, seed=1, learning_rate=1e-3)
    ctx.set_proposal_params(mlp_params(len(ctx.proposal_params()), clusters, 1, 0.3))
    m = ob.OracleMlp(ctx.proposal_params(), cluster_of, clusters, mix=0.9)
    dg, cam = DeviceGBuffer.from_host(g), s.cameras[0].position
    rng = np.random.default_rng(n)
    rows = rng.integers(0, s.width * s.height, n).astype(np.int32)
    targets = rng.integers(0, clusters, n).astype(np.int32)
    targets[5::11] = -1
    targets[-1] = clusters - 1

    def run(r, t):
        return ctx.proposal_gradients(dg, cam, cuda.from_numpy(r).cuda(), cuda.from_numpy(t).cuda())

    grad, loss = run(rows, targets)
    g_gpu = grad.cpu().numpy().astype(np.float64)
    loss_o, g_orc = m.loss_grad(g, cam, rows, targets, emulate=True)
    assert abs(loss - loss_o) <= 1e-4 * abs(loss_o), (loss, loss_o)
    edges = [0, 1024, 1088, 5184, 5248, 9344, 9408, 9408 + 64 * clusters, len(g_orc)]
    for a, b in zip(edges, edges[1:]):
        err = np.linalg.norm(g_gpu[a:b] - g_orc[a:b])
        assert err <= 2e-2 * np.linalg.norm(g_orc[a:b]) + 1e-30, (a, err)
    none, loss0 = run(rows, np.full(n, -1, np.int32))
    assert loss0 == 0.0 and not none.any()
    for k, bad in ((rows, s.width * s.height), (rows, -1), (targets, clusters), (targets, -2)):
        x = k.copy()
        x[-1] = bad
        with pytest.raises(RestirError, match=f"{'row' if k is rows else 'target'} {n - 1} out of range"):
            run(x if k is rows else rows, targets if k is rows else x)
    assert ctx.stats().mma_timeouts == 0
