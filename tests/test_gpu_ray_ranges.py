"""Ray counts on both sides of the lines between the trace kernels' schedules
(csrc/ray_pool.cuh): every form's hits against the oracle, ray by ray."""
import numpy as np
import pytest

import _gpu as G
import _oracle as O
import minimumlbvh_b200 as mb
from minimumlbvh_b200 import scenes

pytestmark = pytest.mark.gpu
LINES = [32, 96, 1024, 1152, 1440, 2016]  # rays per multiprocessor


@pytest.fixture(scope="module")
def scene(cuda):
    tris = scenes.gaussian_soup(700, clusters=6, seed=13)
    b, t, out = G.build(tris)
    w = mb.WideBVH.from_builder(b, t).quantise()
    return tris, b, t, out, w, mb.QuantisedBVH.from_builder(b, t)


@pytest.mark.parametrize("line", LINES)
def test_every_form_at_the_lines(scene, line):
    import torch
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    tris, b, t, out, w, q = scene
    rays = scenes.random_rays(line * sms + 1, tris.reshape(-1, 3).min(0), tris.reshape(-1, 3).max(0), seed=line)
    rays[::13, 4] = 0.0  # the quantised slots' fallback rays
    r = G.dev(rays)
    for query in (0, 1):
        ref = O.trace(out["nodes"], tris, out["root"], rays, query)
        for n in (line * sms - 1, line * sms, line * sms + 1):
            rn = r[:n]
            np.testing.assert_array_equal(G.host(mb.intersect(b, t, rn, query), np.uint32), ref[:n])
            for h in (mb.intersect_wide(w, rn, rayQuery=query),
                      mb.intersect_wide(w, rn, rayQuery=query, quantised=True), mb.intersect_quantised(q, rn, query)):
                h = G.host(h, np.uint32)
                if query == 0:
                    np.testing.assert_array_equal(h, ref[:n])
                else:
                    np.testing.assert_array_equal(h[:, 7] == 0xFFFFFFFF, ref[:n, 7] == 0xFFFFFFFF)
