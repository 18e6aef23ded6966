"""The limit on a walk's steps (2^26, include/mlbvh_device.cuh) counts the
steps that the walk makes: a full walk of a chain of 5.3 million leaves, two
steps a leaf, ends at the chain's end."""
import numpy as np
import pytest

import _gpu as G
import minimumlbvh_b200 as mb

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("query", [mb.RAY_QUERY_CLOSEST, mb.RAY_QUERY_ANY])
def test_long_chain_is_walked_to_its_end(cuda, query):
    import torch
    n = 5_300_000
    leaf = 1 << 31
    # node i: child 0 a leaf of a triangle off the ray, child 1 node i + 1; the last node's child 1 is the one
    # triangle that the ray meets; every box holds the ray
    nodes = torch.zeros((n - 1, 16), dtype=torch.int64, device=cuda)
    i = torch.arange(n - 1, device=cuda)
    nodes[:, 0] = leaf
    nodes[:, 1] = i + 1
    nodes[n - 2, 1] = leaf | 1
    f = np.array([-1, -1, -1, 1, 1, 1] * 2, np.float32).view(np.int32).astype(np.int64)
    nodes[:, 2:14] = torch.from_numpy(f).to(cuda)
    nodes[:, 14] = i - 1
    nodes[:, 15] = -1
    nodes = nodes.to(torch.int32)
    root = torch.zeros(4, dtype=torch.int32, device=cuda)
    tris = G.dev(np.array([[0.5, 0.5, 0, 0.9, 0.5, 0, 0.5, 0.9, 0], [-0.5, -0.5, 0.5, 0.5, -0.5, 0.5, 0, 0.5, 0.5]],
                          np.float32))
    rays = G.dev(np.array([[0, 0, -2, 0, 0, 0, 1, 10]], np.float32))
    hits = G.host(mb.intersect(nodes, tris, rays, query, root=root), np.uint32)
    assert hits[0, 7] == 1 and hits[0, :1].view(np.float32)[0] == 2.5
