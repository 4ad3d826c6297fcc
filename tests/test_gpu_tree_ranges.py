"""The device tree builder at the sizes where its work is divided differently:
around the range that one warp builds whole, around a block's chunk of a big
range, and on leaf orders with long runs of one side (the partition's chains).

Bar: byte-identical to rg_build_bvh, which is byte-identical to the
reference's builder."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _soup(n, seed=5):
    rng = np.random.default_rng(seed)
    c = rng.uniform(-1.0, 1.0, (n, 1, 3))
    return (c + 0.05 * rng.uniform(-1.0, 1.0, (n, 3, 3))).reshape(n, 9).astype(np.float32)


def _same(ctx, cuda, xyz):
    from restir_gb300 import _lib
    n = len(xyz)
    xyz = np.ascontiguousarray(xyz, np.float32)
    hn, ht = np.zeros(n - 1, _lib.NODE_DTYPE), np.zeros(n, _lib.TRI_DTYPE)
    assert _lib.lib().rg_build_bvh(xyz.ctypes.data, n, hn.ctypes.data, ht.ctypes.data) == n - 1
    dev = cuda.from_numpy(xyz).cuda()
    nodes = cuda.full(((n - 1) * 80,), 7, dtype=cuda.uint8, device="cuda")
    tris = cuda.full((n * 48,), 7, dtype=cuda.uint8, device="cuda")
    undef = C.c_int32(-1)
    rc = _lib.lib().rg_build_bvh_device(ctx._h, dev.data_ptr(), n, nodes.data_ptr(), tris.data_ptr(), C.byref(undef),
                                        cuda.cuda.current_stream().cuda_stream)
    assert rc == n - 1, _lib.lib().rg_last_error()
    assert np.array_equal(nodes.cpu().numpy(), hn.view(np.uint8).reshape(-1))
    assert np.array_equal(tris.cpu().numpy(), ht.view(np.uint8).reshape(-1))
    return undef.value


@pytest.mark.parametrize("n", [2, 3, 4, 31, 32, 33, 63, 64, 65, 66, 127, 128, 129, 130, 257, 1023, 1024, 1025, 1089,
                               2049, 4097, 20011, 65537])
def test_sizes(ctx, cuda, n):
    assert _same(ctx, cuda, _soup(n)) == 0


@pytest.mark.parametrize("n", [60, 200, 3000, 50000])
@pytest.mark.parametrize("order", ["descending", "ascending", "few_right_first", "interleaved", "far_outlier"])
def test_leaf_orders(ctx, cuda, n, order):
    xyz = _soup(n, seed=9)
    by_x = np.argsort(xyz[:, 0], kind="stable")
    if order == "descending":
        xyz = xyz[by_x[::-1]]
    elif order == "ascending":
        xyz = xyz[by_x]
    elif order == "few_right_first":  # five leaves of the far side, then the near side in order
        xyz = xyz[np.concatenate([by_x[-5:], by_x[:-5]])]
    elif order == "interleaved":
        xyz = xyz[np.concatenate([by_x[::-2], by_x[::2] if n % 2 else by_x[0::2]])]
    else:  # one side of every split is tiny: a deep, uneven tree
        xyz = xyz * (np.float32(2.0) ** -np.linspace(0, 60, n, dtype=np.float32))[:, None]
    _same(ctx, cuda, xyz)


@pytest.mark.parametrize("n", [40, 100, 3000])
def test_median_splits(ctx, cuda, n):
    """Equal centroids (every split the median one) beside distinct ones, at sizes of one warp and of blocks."""
    one = np.repeat(_soup(1), n, axis=0)
    assert _same(ctx, cuda, one) == 1
    assert _same(ctx, cuda, np.concatenate([_soup(n), one, np.repeat(_soup(2, seed=3), n, axis=0)])) == 1


def test_workspace_is_reused_across_sizes(ctx, cuda):
    for n in (5000, 100, 40000, 65, 5000):
        assert _same(ctx, cuda, _soup(n, seed=n)) == 0
