"""Builds back to back on one stream with one scratch, each kernel starting
while the one before it drains (csrc/chain.cuh): every build is of its own
scene, launched directly or replayed from a captured graph."""
import numpy as np
import pytest

import _gpu as G
import _oracle as O
import minimumlbvh_b200 as mb
from minimumlbvh_b200 import scenes

pytestmark = pytest.mark.gpu
SIZES = [1000, 4096, 4097, 20000, 120000, 460000]  # one-CTA sort, small and large sort tiles, tile groups


def two_scenes(n):
    tris = [scenes.gaussian_soup(n, clusters=8, seed=s) for s in (31, 32)]
    return tris, [O.build(t) for t in tris]


def check(nodes, root, ref):
    np.testing.assert_array_equal(G.host(nodes, np.uint32)[: len(ref["nodes"])], ref["nodes"])
    assert int(G.host(root, np.uint32)[0]) == ref["root"]


@pytest.mark.parametrize("n", SIZES)
def test_alternating_scenes(cuda, n):
    import torch
    tris, refs = two_scenes(n)
    t = [G.dev(x) for x in tris]
    sorter, b = mb.OnesweepSort(), mb.BVHGPUBuilder()
    kept = []
    for i in range(8):
        b.build(t[i % 2], n, 0, sorter)
        kept.append((b.m_internals.clone(), b.m_rootNode.clone()))
    b.status()
    for i, (nodes, root) in enumerate(kept):
        check(nodes, root, refs[i % 2])


@pytest.mark.parametrize("n", SIZES)
def test_captured_build(cuda, n):
    import torch
    tris, refs = two_scenes(n)
    t = [G.dev(x) for x in tris]
    inp = t[0].clone()
    sorter, b = mb.OnesweepSort(), mb.BVHGPUBuilder()
    b.build(inp, n, 0, sorter)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        b.build(inp, n, 0, sorter)
    for i in (1, 0, 1):
        inp.copy_(t[i])
        b.m_internals.fill_(-1)
        g.replay()
        b.status()
        check(b.m_internals, b.m_rootNode, refs[i])
