"""The tiled tree build (csrc/tree.cuh) against the oracle, bit for bit, where
its tiles (256 leaves), groups (32 tiles) and supers (32 groups) begin and
end, where runs of equal keys cross tiles, and where it hands the build to
the leaf-by-leaf climb: NaN centroids, and too many crossing nodes."""
import numpy as np
import pytest

import _gpu as G
import _oracle as O
import minimumlbvh_b200 as mb
from minimumlbvh_b200 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [254, 511, 512, 513, 769, 8192, 8193, 8449, 262144, 262145, 262400, 530001])
def test_tile_group_and_super_edges(cuda, n):
    tris = scenes.gaussian_soup(n, clusters=16, seed=40 + n)
    _, _, out = G.build(tris)
    G.assert_build_equal(out, O.build(tris))


@pytest.mark.parametrize("run", [2, 31, 255, 256, 257, 600])
def test_runs_of_equal_keys_across_tiles(cuda, run):
    """Runs short and long beside 20,000 other triangles: records for the few
    crossing nodes, the climb where runs make too many."""
    tris = np.concatenate([scenes.gaussian_soup(20000, clusters=8, seed=run),
                           np.repeat(scenes.gaussian_soup(max(1, 1800 // run), clusters=8, seed=run + 1), run, 0)])
    _, _, out = G.build(tris)
    G.assert_build_equal(out, O.build(tris))


def _tree_of_keys(out, tris):
    """The oracle's tree over the GPU's sorted keys (bounds of scenes with
    NaN depend on the platform's minimum, and the keys with them)."""
    n = len(tris)
    nodes, deltas, root = np.zeros((n - 1, 16), np.uint32), np.zeros(n - 1, np.uint8), np.zeros(1, np.uint32)
    tris = np.ascontiguousarray(tris, np.float32)
    O.oracle().orc_build_from_keys(O.P(out["keys"].copy()), O.P(out["indices"].copy()), O.P(tris), n, O.P(nodes),
                                   O.P(deltas), O.P(root))
    return nodes, int(root[0])


@pytest.mark.parametrize("n,step", [(300, 299), (5000, 97), (40000, 39999)])
def test_nan_vertices_take_the_climb(cuda, n, step):
    tris = scenes.gaussian_soup(n, clusters=4, seed=n)
    tris[::step, 7] = np.nan
    _, _, out = G.build(tris)
    nodes, root = _tree_of_keys(out, tris)
    np.testing.assert_array_equal(out["nodes"], nodes)
    assert out["root"] == root


def test_signed_zeros_and_infinities(cuda):
    rng = np.random.default_rng(3)
    tris = rng.random((9000, 3, 3)).astype(np.float32) - np.float32(0.5)
    tris[rng.random(tris.shape) < 0.2] = 0.0
    tris[rng.random(tris.shape) < 0.2] = -0.0
    flat = tris.reshape(-1, 9).copy()
    _, _, out = G.build(flat)
    G.assert_build_equal(out, O.build(flat))
    flat[17, 4] = np.inf  # an infinite extent: the axis's keys are conversions of NaN or 0
    _, _, out = G.build(flat)
    np.testing.assert_array_equal(out["nodes"], _tree_of_keys(out, flat)[0])


@pytest.mark.parametrize("nan", [False, True])
def test_batched_meshes_end_at_tile_edges(cuda, nan):
    import torch
    sizes = [256, 1, 255, 1, 1, 300, 212, 512, 2, 254, 9000, 1, 257, 255]
    off = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int64)
    tris = np.concatenate([scenes.gaussian_soup(k, clusters=3, seed=70 + i) for i, k in enumerate(sizes)])
    if nan:
        tris[off[10] + 5, 1] = np.nan
    b = mb.BatchedBVH(G.dev(tris), G.dev(off.astype(np.int32)), len(sizes)).build()
    b.status()
    nodes, roots = G.host(b.internals, np.uint32), G.host(b.roots, np.uint32)
    for m, k in enumerate(sizes):
        mesh = tris[off[m]:off[m + 1]]
        ref = G.build(mesh)[2] if np.isnan(mesh).any() else O.build(mesh)
        assert roots[m] == ref["root"], m
        np.testing.assert_array_equal(nodes[off[m] - m: off[m + 1] - m - 1], ref["nodes"], err_msg=f"mesh {m}")
