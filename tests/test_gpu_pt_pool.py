"""The path tracer's pixel pool: images of one pixel, of partial 8 x 4 tiles
and of several tiles per CTA, both sample streams, depth and sample limits,
against the oracle's pt bit for bit."""
import numpy as np
import pytest

import _gpu as G
import _oracle as O
import minimumlbvh_b200 as mb
from minimumlbvh_b200 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h,sobol,depth,spp", [(1, 1, 1, 1024, 9), (9, 5, 0, 1024, 9), (31, 3, 1, 0, 9),
                                                 (33, 130, 1, 1, 9), (613, 401, 1, 4, 1), (250, 97, 0, 3, 2)])
def test_pt_pool_edges(cuda, w, h, sobol, depth, spp):
    import torch
    tris = scenes.heightfield_icospheres(seed=4, quads=48, spheres=6, level=2)
    b, t, out = G.build(tris)
    attribs = scenes.pt_attributes(len(tris), light_fraction=0.05)
    cam = O.lookat(*scenes.camera_heightfield(), w, h)
    acc = torch.zeros((w * h, 4), dtype=torch.float32, device="cuda")
    ref = np.zeros((w * h, 4), np.float32)
    lt = mb.leaf_triangles(b, t)
    for k in range(3):
        mb.render_pt(acc, (w, h), mb.RayGenerator.from_array(cam), b.m_rootNode, b.m_internals, t, G.dev(attribs),
                     sobol, spp, depth, traversal=mb.TRAVERSAL_REPLAY if k == 1 else mb.TRAVERSAL_STACKFREE,
                     leaf_triangles=lt if k == 1 else None)
        O.render_pt(ref, cam, out["root"], out["nodes"], tris, attribs, w, h, sobol, spp, depth,
                    trig=1)
    np.testing.assert_array_equal(G.host(acc), ref)
