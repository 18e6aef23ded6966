"""Differentiable renders whose warps draw samples from units of pixels: units
that hold many pixels, a part of one, and a single pixel, against the oracle's
FP32 image bit for bit."""
import numpy as np
import pytest

import _gpu as G
import _oracle as O
import minimumlbvh_b200 as mb
from minimumlbvh_b200 import scenes

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def scene(cuda):
    tris, alb, em = scenes.diff_scene()
    b, t, out = G.build(tris)
    return tris, alb, em, b, t, out


@pytest.mark.parametrize("w,h,spp", [(211, 101, 1), (160, 140, 5), (150, 80, 65), (33, 9, 130), (1, 1, 200)])
def test_diff_render_units_and_pixel_ranges(scene, w, h, spp):
    """Warps that take several pixels, units of 64 samples that hold many
    pixels or a part of one, and a single pixel."""
    import torch
    tris, alb, em, b, t, out = scene
    eye, c, up, fovy = scenes.camera_heightfield()
    cam = mb.RayGenerator().lookat(eye, c, up, fovy, w, h)
    img = torch.empty(w * h, dtype=torch.float32, device="cuda")
    mb.pt_diff_render(img, (w, h), cam, b, t, G.dev(alb), G.dev(em), spp, 2)
    np.testing.assert_array_equal(G.host(img), O.diff_render(out, tris, cam.as_array(), w, h, spp, 2, alb, em))
