"""Builds that the range queries leave to the climb (csrc/climb.cuh), beyond one
round of its resident CTAs (303,104 leaves), and batches of meshes so small
that their trees' ends outnumber the records."""
import numpy as np
import pytest

import _gpu as G
import _oracle as O
import minimumlbvh_b200 as mb
from minimumlbvh_b200 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [8192, 8193, 303_104, 303_200, 700_001])
def test_runs_of_equal_keys(cuda, n):
    run = 40
    tris = np.repeat(scenes.gaussian_soup((n + run - 1) // run, clusters=8, seed=n), run, 0)[:n]
    tris = np.concatenate([tris[: n // 2], np.repeat(tris[n // 2: n // 2 + 1], 900, 0), tris[n // 2:]])[:n]
    _, _, out = G.build(tris)
    G.assert_build_equal(out, O.build(tris))


@pytest.mark.parametrize("meshes", [40, 700, 3000, 50_000])
def test_batches_of_tiny_meshes(cuda, meshes):
    sizes = np.random.default_rng(meshes).integers(1, 17, meshes)
    off = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int64)
    tris = scenes.gaussian_soup(int(off[-1]), clusters=40, seed=meshes)
    b = mb.BatchedBVH(G.dev(tris), G.dev(off.astype(np.int32)), meshes).build()
    b.status()
    nodes, roots = G.host(b.internals, np.uint32), G.host(b.roots, np.uint32)
    for m in range(0, meshes, max(1, meshes // 500)):
        ref = O.build(tris[off[m]:off[m + 1]])
        assert roots[m] == ref["root"], m
        np.testing.assert_array_equal(nodes[off[m] - m: off[m + 1] - m - 1], ref["nodes"], err_msg=f"mesh {m}")
