"""How the differentiable kernels share an image out: a warp per pixel in small
images of few samples (up to 52 pixels and 256 samples per multiprocessor, 108
pixels and 16 samples in views at least 2.5 times as wide as high), else groups
of pixels all over the image, single pixels of many samples or in wide views;
strides that would fall into the same columns, partial last groups. The image
against the oracle's bit for bit, the gradient against its FP64 adjoint (1e-3
relative, as test_gpu_adjoint.py, at triangles with at least 1 % of the
largest)."""
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


@pytest.mark.parametrize("w,h,spp", [(64, 74, 8), (64, 74, 9), (149, 32, 8), (1, 1, 3), (300, 40, 4), (401, 61, 2),
                                     (400, 60, 64), (512, 32, 33), (201, 201, 5), (131, 97, 1), (104, 74, 4),
                                     (105, 74, 4), (50, 63, 12), (50, 63, 13), (216, 74, 16), (217, 74, 16),
                                     (216, 74, 17), (101, 67, 24), (101, 67, 23), (260, 113, 3)])
def test_image_and_gradient(scene, w, h, spp):
    import torch
    tris, alb, em, b, t, out = scene
    eye, c, up, fovy = scenes.camera_heightfield()
    cam = mb.RayGenerator().lookat(eye, c, up, fovy, w, h)
    img = torch.full((w * h,), -1.0, dtype=torch.float32, device="cuda")
    args = ((w, h), cam, b, t, G.dev(alb), G.dev(em), spp, 2)
    mb.pt_diff_render(img, *args)
    np.testing.assert_array_equal(G.host(img), O.diff_render(out, tris, cam.as_array(), w, h, spp, 2, alb, em))
    weight = np.random.default_rng(w).uniform(0.5, 1.5, w * h).astype(np.float32)
    grad = torch.zeros(len(tris), dtype=torch.float32, device="cuda")
    mb.pt_diff_adjoint(grad, G.dev(weight), *args)
    host = O.diff_adjoint(out, tris, cam.as_array(), w, h, spp, 2, alb, em, weight.astype(np.float64))
    big = np.abs(host) > 0.01 * np.abs(host).max()
    np.testing.assert_allclose(G.host(grad)[big], host[big], rtol=1e-3)
