"""The tree builder's workspace is kept between builds and given back by the
next scene upload."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_upload_gives_the_workspace_back(cuda, restir_lib):
    from restir_gb300 import _lib, scenes
    from restir_gb300.passes import Context
    n = 1 << 20
    s = scenes.config2(width=16, height=16, n_tris=1000, n_lights=64, frames=1)
    ctx = Context(0)
    try:
        ctx.upload_scene(s)
        xyz = cuda.rand((n, 9), dtype=cuda.float32, device="cuda")
        nodes = cuda.empty(((n - 1) * 80,), dtype=cuda.uint8, device="cuda")
        tris = cuda.empty((n * 48,), dtype=cuda.uint8, device="cuda")

        def build():
            rc = _lib.lib().rg_build_bvh_device(ctx._h, xyz.data_ptr(), n, nodes.data_ptr(), tris.data_ptr(), None,
                                                cuda.cuda.current_stream().cuda_stream)
            assert rc == n - 1, _lib.lib().rg_last_error()
            cuda.cuda.synchronize()
            return cuda.cuda.mem_get_info()[0], nodes.cpu().numpy()

        cuda.cuda.synchronize()
        _, first = build()          # the code's own first-use allocations
        ctx.upload_scene(s)
        before = cuda.cuda.mem_get_info()[0]
        held, again = build()
        assert before - held > 150 * n and np.array_equal(first, again)
        assert build()[0] == held   # a repeated build allocates nothing
        ctx.upload_scene(s)
        assert cuda.cuda.mem_get_info()[0] >= before - (8 << 20)
        assert np.array_equal(build()[1], first)
    finally:
        ctx.close()
