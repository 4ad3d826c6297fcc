"""Learned-proposal inference with one to four chunks of 64 clusters (the ring
of three bias tiles before, at and after its first reuse), a ragged last row
tile and the fewest and most candidates, against the oracle.

Tolerances: one hidden value on the other side of a bf16 rounding boundary
(2^-8 relative) moves a logit by at most 2^-8 |h| |w| < 2e-3 here, and with it
the log-sum-exp; a candidate's probability by the same relative amount plus
that of the log-sum-exp, below 1e-2; and its cluster only where a uniform lies
within such a step of an interval's end, below one in two hundred.
"""
from __future__ import annotations

import numpy as np
import pytest

import oracle_binding as ob
from helpers import mlp_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("clusters", [64, 128, 192, 256])
@pytest.mark.parametrize("n_cand", [1, 32])
def test_inference_at_chunk_counts(ctx, cuda, restir_lib, clusters, n_cand):
    from restir_gb300 import _lib, scenes
    from restir_gb300.passes import DeviceGBuffer
    s = scenes.config2(width=61, height=47, n_tris=2000, n_lights=1024, frames=1)
    g = scenes.trace_gbuffer_host(s, 0)
    cluster_of = (np.arange(len(s.point_lights)) % clusters).astype(np.int32)
    ctx.upload_scene(s)
    ctx.create_proposal(cluster_of, clusters, mix=0.9, batch=256, seed=1, learning_rate=1e-3)
    ctx.set_proposal_params(mlp_params(len(ctx.proposal_params()), clusters, 2, 0.3))
    m = ob.OracleMlp(ctx.proposal_params(), cluster_of, clusters, mix=0.9)
    u = s.uniforms(0)
    u.flags |= _lib.RG_FLAG_LEARNED_PROPOSAL
    u.initial_light_sample_count = n_cand
    n = s.width * s.height
    ctx.proposal_infer(DeviceGBuffer.from_host(g), u)
    cand, stat = ctx.proposal_buffers(n)
    lse, _ = m.row_stats(g, s.cameras[0].position)
    assert np.abs(stat[:, 0].astype(np.float64) - lse).max() <= 2e-3
    keys, qs = m.sample(g, s.cameras[0].position, u.frame, n_cand, np.arange(n, dtype=np.int32))
    got_k, got_q = cand["key"][:, :n_cand], cand["q"][:, :n_cand]
    uni = keys >= 0
    assert np.array_equal(got_k >= 0, uni)
    assert np.array_equal(got_k[uni], keys[uni])
    same = got_k == keys
    assert same[~uni].mean() >= 0.995, same[~uni].mean()
    rel = np.abs(got_q[same] - qs[same]) / np.maximum(qs[same], 1e-30)
    assert rel.max() <= 1e-2, rel.max()
    assert ctx.stats().mma_timeouts == 0
