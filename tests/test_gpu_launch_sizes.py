"""Batches of shadow segments and RIS frames at the sizes where their launch
shape changes, and the G-buffer of cameras whose rays leave the packed slab test.

Bar: bit-exact.  A segment's answer does not depend on its batch (the large
batch is pinned against the oracle in test_gpu_visibility.py); G-buffer planes
equal the library's CPU tracer byte for byte."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def scene(restir_lib):
    from restir_gb300 import scenes
    return scenes.config2(width=64, height=64, n_tris=5000, n_lights=64, frames=1)


def test_batch_sizes(ctx, cuda, scene):
    ctx.upload_scene(scene)
    rng = np.random.default_rng(3)
    big = 700_000
    p = [np.concatenate([rng.uniform(0.0, 1.0, (big, 3)), np.ones((big, 1))], 1).astype(np.float32) for _ in range(2)]
    t1, t2 = (cuda.from_numpy(a).cuda() for a in p)
    ref = cuda.full((big,), 9, dtype=cuda.uint8, device="cuda")
    ctx.visibility_batch(t1, t2, ref)
    assert int(ref.max()) == 1 and int(ref.min()) == 0
    edge = 1216 * 32
    for n in (1, 2, 3, 4, 5, 31, 33, 129, 2003, 4 * 1216, 4 * 1216 + 1, edge - 1, edge, edge + 1, 152 * 8 * 128,
              152 * 8 * 128 + 1, 152 * 8 * 512 - 1, 152 * 8 * 512 + 1):
        out = cuda.full((n + 1,), 9, dtype=cuda.uint8, device="cuda")
        ctx.visibility_batch(t1[:n], t2[:n], out)
        assert cuda.equal(out[:n], ref[:n]) and int(out[n]) == 9, n


@pytest.mark.parametrize("size", [(1, 1), (17, 9), (33, 33), (65, 7)])
@pytest.mark.parametrize("target", [(0.5, 0.5, 0.9), (0.9, 0.5, 0.5), (0.1, 0.5, 0.5), (0.52, 0.47, 0.9)])
def test_gbuffer_of_axis_aligned_cameras(ctx, cuda, scene, size, target):
    from restir_gb300 import scenes
    from restir_gb300.camera import CameraModel
    from restir_gb300.passes import DeviceGBuffer
    w, h = size
    cam = CameraModel(position=np.array([0.5, 0.5, 0.5], np.float32), look_at=np.array(target, np.float32), aspect=w / h)
    s = scene.view(cam, w, h)
    ctx.upload_scene(s)
    g = DeviceGBuffer(w, h)
    ctx.trace_gbuffer(cam, g)
    host = scenes.trace_gbuffer_host(s, 0)
    dev = g.to_host()
    for k, v in host.items():
        assert np.array_equal(v.view(np.uint8), dev[k].view(np.uint8)), k


@pytest.mark.parametrize("samples,mis", [(1, 0), (1, 1), (2, 0), (2, 1)])
@pytest.mark.parametrize("rows", [1, 100, 310, 311])
def test_ris_frames_on_both_sides_of_the_shape_rule(ctx, cuda, scene, samples, mis, rows):
    """A pixel's RIS result depends on its coordinates and texel only, so the
    top rows of a frame just above the rule's pixel count (several pixels per
    thread) equal those of a frame with only these rows (one per thread)."""
    from restir_gb300.passes import DeviceGBuffer, reservoirs
    w, h = 501, 313
    assert w * 310 < 152 * 8 * 128 < w * 311
    s = scene.view(scene.cameras[0], w, h)
    ctx.upload_scene(s)
    ctx.set_reservoir_format(samples, mis)
    try:
        nbytes = ctx.reservoir_bytes()
        g = DeviceGBuffer(w, h)
        ctx.trace_gbuffer(s.cameras[0], g)
        u = s.uniforms(0)
        full = reservoirs(w * h, nbytes=nbytes)
        ctx.initial_temporal(g, None, None, full, u)
        top = DeviceGBuffer(w, rows)
        for k, t in top.planes.items():
            t.copy_(g.planes[k][:rows])
        u.screen_size[:] = [w, rows]
        part = reservoirs(w * rows, nbytes=nbytes)
        ctx.initial_temporal(top, None, None, part, u)
        assert cuda.equal(part, full[:w * rows])
        assert int((full != 0).sum()) > 0
    finally:
        ctx.set_reservoir_format(1, 0)


def test_reservoir_buffers_at_16_byte_alignment(ctx, cuda, scene):
    """The spatial and shading passes read reservoirs by 256-bit loads where
    the buffer is 32-byte aligned; a caller's need only be 16-byte aligned."""
    from restir_gb300.passes import DeviceGBuffer, reservoirs
    w, h = 77, 45
    s = scene.view(scene.cameras[0], w, h)
    ctx.upload_scene(s)
    g = DeviceGBuffer(w, h)
    ctx.trace_gbuffer(s.cameras[0], g)
    u = s.uniforms(0)
    n = w * h
    r0 = reservoirs(n)
    ctx.initial_temporal(g, None, None, r0, u)
    raw = cuda.zeros(n * 16 + 4, dtype=cuda.int32, device="cuda")
    shifted = raw[4:].view(n, 16)
    shifted.copy_(r0)
    assert r0.data_ptr() % 32 == 0 and shifted.data_ptr() % 32 == 16
    outs = []
    for src in (r0, shifted):
        ctx.initial_temporal(g, None, None, reservoirs(n), u)
        a, b = reservoirs(n), reservoirs(n)
        ctx.spatial_unbiased(g, src, a, u, 5, 0)
        ctx.spatial_biased(g, src, b, u, 0)
        img = cuda.zeros((h, w, 4), dtype=cuda.float32, device="cuda")
        ctx.shade(g, src, s.lighting_uniforms(0), img)
        outs.append((a, b, img.view(cuda.int32)))
    for p, q in zip(*outs):
        assert cuda.equal(p, q)
