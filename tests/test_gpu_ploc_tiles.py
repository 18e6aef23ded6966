"""PLOC builds at the edges of both tile sizes of the grid phase against the
oracle, node by node: small tiles (256 - 2r clusters each, up to 151,552
clusters) past the one-CTA tail, large ones (1,024 - 2r) above, the change from
large to small, every compiled radius, and equal boxes (hashed ties, pairing)."""
import numpy as np
import pytest

import _gpu as G
import _oracle as O
import minimumlbvh_b200 as mb
from minimumlbvh_b200 import scenes

pytestmark = pytest.mark.gpu


def check(tris, radius):
    n = len(tris)
    b = mb.BVHGPUBuilder().buildByPLOC(G.dev(np.ascontiguousarray(tris, np.float32).reshape(-1, 9)), n, 0, None, radius)
    b.status()
    ref = O.build_ploc(tris, 0, radius)
    assert int(G.host(b.m_rootNode, np.uint32)[0]) == ref["root"]
    bad = np.nonzero((G.host(b.m_internals, np.uint32)[: n - 1] != ref["nodes"]).any(1))[0]
    assert bad.size == 0, f"{bad.size} nodes differ, first {bad[:5]}"


@pytest.mark.parametrize("radius", [1, 4, 8, 16, 32])
@pytest.mark.parametrize("tiles,more", [(6, 0), (6, 1), (9, 0), (9, 1)])
def test_small_tiles(cuda, radius, tiles, more):
    check(scenes.gaussian_soup(tiles * (256 - 2 * radius) + more, clusters=4, seed=radius), radius)


@pytest.mark.parametrize("radius", [1, 4, 7, 8, 16, 32])
@pytest.mark.parametrize("n", [151_552, 151_553, 0, 1])
def test_large_tiles(cuda, radius, n):
    if n < 2:  # whole large tiles, and one cluster more
        tile = 1024 - 2 * radius
        n += (151_553 + tile - 1) // tile * tile
    check(scenes.gaussian_soup(n, clusters=16, seed=radius), radius)


@pytest.mark.parametrize("radius", [1, 8, 32])
def test_equal_boxes_in_large_tiles(cuda, radius):
    check(np.tile(scenes.gaussian_soup(4, clusters=2, seed=3), (40_000, 1)), radius)
