"""Ray counts at the edges of the pooled trace kernels' blocks (8 and 32 rays),
of one CTA per multiprocessor pair, and past one block per resident CTA: every
form's hits against the oracle's stack-free walk, ray by ray."""
import numpy as np
import pytest

import _gpu as G
import _oracle as O
import minimumlbvh_b200 as mb
from minimumlbvh_b200 import scenes

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def scene(cuda):
    tris = scenes.gaussian_soup(3000, clusters=6, seed=12)
    b, t, out = G.build(tris)
    w = mb.WideBVH.from_builder(b, t).quantise()
    return tris, b, t, out, w, mb.QuantisedBVH.from_builder(b, t)


@pytest.mark.parametrize("n", [1, 7, 8, 9, 33, 2367, 2369, 9473, 37889, 151_590])
def test_every_form_at_pool_edges(scene, n):
    tris, b, t, out, w, q = scene
    rays = scenes.random_rays(n, tris.reshape(-1, 3).min(0), tris.reshape(-1, 3).max(0), seed=n)
    rays[::13, 4] = 0.0  # the quantised slots' fallback rays
    r = G.dev(rays)
    for query in (0, 1):
        ref = O.trace(out["nodes"], tris, out["root"], rays, query)
        hits = G.host(mb.intersect(b, t, r, query), np.uint32)
        np.testing.assert_array_equal(hits, ref)
        forms = [mb.intersect_wide(w, r, rayQuery=query), mb.intersect_wide(w, r, rayQuery=query, quantised=True),
                 mb.intersect_quantised(q, r, query)]
        for h in forms:
            h = G.host(h, np.uint32)
            if query == 0:
                np.testing.assert_array_equal(h, ref)
            else:
                np.testing.assert_array_equal(h[:, 7] == 0xFFFFFFFF, ref[:, 7] == 0xFFFFFFFF)
