"""The split deltas of mlbvh_build_ex for scenes with NaN vertices, whose
trees are climbed leaf by leaf (csrc/tree.cuh): written for every build, as the
sorted keys fix them."""
import numpy as np
import pytest

import _gpu as G
import _oracle as O
import minimumlbvh_b200 as mb
from minimumlbvh_b200 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,step", [(2, 1), (300, 299), (5000, 97), (40000, 39999)])
def test_deltas_with_nan_vertices(cuda, n, step):
    import torch
    tris = scenes.gaussian_soup(max(n, 8), clusters=4, seed=n)[:n].copy()
    tris[::step, 7] = np.nan
    t = G.dev(tris)
    L = mb.lib()
    nodes = torch.empty((n, 16), dtype=torch.int32, device=cuda)
    root = torch.empty(4, dtype=torch.int32, device=cuda)
    keys, idx = (torch.empty(n, dtype=torch.int32, device=cuda) for _ in range(2))
    deltas = torch.full((max(n, 16),), 0xEE, dtype=torch.uint8, device=cuda)  # no delta has this value
    scratch = torch.empty(L.mlbvh_build_scratch_bytes(n), dtype=torch.uint8, device=cuda)
    stream = torch.cuda.current_stream().cuda_stream
    assert L.mlbvh_build_ex(t.data_ptr(), n, 0, nodes.data_ptr(), root.data_ptr(), None, keys.data_ptr(),
                            idx.data_ptr(), deltas.data_ptr(), scratch.data_ptr(), scratch.numel(), stream) == 0
    assert L.mlbvh_scratch_status(scratch.data_ptr(), stream) == 0
    ref_nodes, ref, ref_root = np.zeros((n - 1, 16), np.uint32), np.zeros(n - 1, np.uint8), np.zeros(1, np.uint32)
    O.oracle().orc_build_from_keys(O.P(G.host(keys, np.uint32).copy()), O.P(G.host(idx, np.uint32).copy()),
                                   O.P(np.ascontiguousarray(tris, np.float32)), n, O.P(ref_nodes), O.P(ref),
                                   O.P(ref_root))
    np.testing.assert_array_equal(G.host(nodes, np.uint32)[: n - 1], ref_nodes)
    got = G.host(deltas)
    np.testing.assert_array_equal(got[: n - 1], ref)
    assert (got[n:] == 0xEE).all()
