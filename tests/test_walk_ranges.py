"""The quantized walk's range of scenes and segments.

Every scene that the packing takes gets the quantized copy, and every segment
that the filtered slab test takes (components within 2^+-100) walks it, unless
its smallest component is below 2^-120 of the scene's and origin's magnitude
(rgm::walk_fits).  On the CPU (tests/walk_range_check.cu): the planes'
distances stay finite and the walk tests the reference's triangles.  On the
GPU: the layout in use, and answers equal to the oracle's bit for bit, on both
sides of that limit."""
from __future__ import annotations

import ctypes as C
import dataclasses
import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

ROOT = Path(__file__).resolve().parents[1]
CSRC = ROOT / "restir-vulkan_gb300" / "csrc"


@pytest.fixture(scope="module")
def checker(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not Path(nvcc).exists():
        pytest.skip("nvcc not found")
    exe = tmp_path_factory.mktemp("walk") / "walk_range_check"
    cmd = [nvcc, "-std=c++17", "-O2", "-Xcompiler", "-ffp-contract=off,-fopenmp", f"-I{CSRC}",
           str(ROOT / "tests" / "walk_range_check.cu"), str(CSRC / "host.cpp"), "-o", str(exe), "-lgomp"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-3000:]
    return exe


@pytest.mark.parametrize("scale", [-100, -60, -20, 0, 27, 31, 33, 64, 100])
def test_every_magnitude_walks_the_copy(checker, scale):
    r = subprocess.run([str(checker), str(scale), "3000"], capture_output=True, text=True, timeout=600)
    print(r.stdout)
    assert r.returncode == 0, r.stdout + r.stderr
    f = dict(zip(r.stdout.split()[0::2], r.stdout.split()[1::2]))
    assert f["containment_failures"] == "0" and f["infinite"] == "0"
    assert f["set_mismatches"] == "0" and f["answer_mismatches"] == "0"
    assert f["fast"] == f["usable"] and int(f["usable"]) > 500
    if -30 < scale < 40:  # beyond, the reference's triangle test answers no
        assert 0.2 < int(f["hits"]) / int(f["usable"]) < 0.9


@pytest.mark.gpu
@pytest.mark.parametrize("scale", [-40, -20, 0, 20, 31, 33, 40, 60])
def test_scaled_scene_bit_exact(ctx, cuda, oracle_lib, restir_lib, scale):
    """A scene scaled by a power of two, which keeps its tree: random segments,
    segments with one component from 2^-10 to 2^-125 of the scene (past
    2^-100, and past 2^-120 of a large scene, they leave the copy) and segments
    from 2^10 to 2^45 scene sizes away."""
    from restir_gb300 import scenes
    ob = oracle_lib
    s = scenes.config1()
    f = np.float32(2.0) ** np.float32(scale)
    nodes, tris = s.nodes.copy(), s.triangles.copy()
    for a in (nodes, tris):
        for k in a.dtype.names:
            if a.dtype[k].base == np.float32:
                a[k][..., :3] *= f
    s = dataclasses.replace(s, nodes=nodes, triangles=tris)
    rng = np.random.default_rng(5)
    n = 30_000
    lo = np.minimum(nodes["lmin"][0, :3], nodes["rmin"][0, :3]) / f
    hi = np.maximum(nodes["lmax"][0, :3], nodes["rmax"][0, :3]) / f
    p = [(lo + (hi - lo) * rng.uniform(0.0, 1.0, (n, 3))).astype(np.float32) for _ in range(2)]
    third = n // 3
    tiny, ax = np.arange(third), rng.integers(0, 3, third)
    p[0][tiny, ax] = 0.0
    p[1][tiny, ax] = np.ldexp(np.float32(1.0), -rng.integers(10, 126, third)).astype(np.float32)
    far = np.arange(third, 2 * third)
    away = np.ldexp(1.0, rng.integers(10, 46, third))[:, None]
    step = rng.uniform(-1.0, 1.0, (third, 3))
    mid = p[1][far].astype(np.float64)
    p[0][far], p[1][far] = (mid + away * step).astype(np.float32), (mid - step).astype(np.float32)
    ends = [np.ascontiguousarray(a * f) for a in p]
    ctx.upload_scene(s)
    out = cuda.full((n,), 9, dtype=cuda.uint8, device="cuda")
    ctx.stats(reset=True)
    ctx.visibility_batch(*(cuda.from_numpy(np.concatenate([a, np.ones((n, 1), np.float32)], 1)).cuda() for a in ends), out)
    st = ctx.stats()
    assert st.traversal_errors == 0 and st.tree_layout == ctx.TREE_LAYOUTS["quant"]
    exp = np.zeros(n, np.uint8)
    sc, keep = ob.scene_struct(s)
    ob.oracle().or_test_visibility_batch(C.byref(sc), n, ob.P(ends[0]), ob.P(ends[1]), ob.P(exp), None)
    got = out.cpu().numpy()
    assert np.array_equal(got, exp), f"{np.count_nonzero(got != exp)} of {n} bits differ"
    if abs(scale) <= 20:
        assert 0.02 < exp.mean() < 0.98
