"""Rounding of the adjoint's 32-bit sums: a gradient against the 64-bit sum of the
gradients of the image's bands (dL/dI zero outside the band), whose sums are
shorter by the number of bands.

Terms go through three levels of sums: n1 in a block's first array, n2 of those
in its second, 148 blocks' in the gradient.  A running sum of n like terms rounds
by about sqrt(n) / 6 units of 2^-24 (rms); the errors of the independent sums of
one level average out in the next.  At 512x512, 8 bounces, with 8 lanes of 4
samples: n1 about 256 lanes x 4 samples x 2 vertices, n2 55, so sqrt(2048) / 6
/ sqrt(55 x 148) + sqrt(55) / 6 / sqrt(148) + sqrt(148) / 6 = 2.2 units; 8 units
are the bound.  With equal terms, as of an emitter that fills the frame,
the roundings add up instead: n / 2 units a level, (256 x 2 + 14) / 2 + 148 / 2."""
import numpy as np
import pytest

from raymotion_b200 import RenderConfig, _abi
from raymotion_b200.scene import Camera
from raymotion_b200.scenes import PLAIN_FLAGS, inverse_scene

from . import kat_scenes as K
from .test_gpu_adjoint import _grad, _set, _torch

pytestmark = pytest.mark.gpu


def test_gradient_against_bands_summed_in_64_bits(backend):
    torch = _torch()
    w = 512
    d = inverse_scene(4, n_spheres=20, n_dielectric=6, ground=40, width=w, height=w, spp=32, depth=8)
    n = w * w * 3
    dl = torch.rand(n, device="cuda", generator=torch.Generator("cuda").manual_seed(1)) * (2.0 / n)
    h = backend.scene_create(d["scene"])
    try:
        _set(backend, h, d, d["params"])
        want = 0.0
        for band in range(32):
            part = torch.zeros_like(dl)
            part[band * n // 32:(band + 1) * n // 32] = dl[band * n // 32:(band + 1) * n // 32]
            want = want + _grad(backend, h, d, 5, part).astype(np.float64)
        got = _grad(backend, h, d, 5, dl).astype(np.float64)
    finally:
        backend.scene_destroy(h)
    err = np.linalg.norm(got - want) / np.linalg.norm(want)
    assert err <= 8 * 2.0 ** -24, err


@pytest.mark.parametrize("value", [0.1, 0.3, 0.7, 0.9])
def test_equal_terms(backend, value):
    torch = _torch()
    w, spp = 256, 8
    sc = K.fullscreen_emitter()
    cam = Camera()
    cam.focal = w * 0.866
    cam.update_trig()
    cfg = RenderConfig(width=w, height=w, spp=spp, max_bounces=1, restir_candidates=1, restir_spatial=0, adapt_min=0,
                       flags=PLAIN_FLAGS | _abi.RM_FLAG_NOADAPT)
    prm = np.array([[1, 1, 1, 0.5, 1, 0, 0, 1]], np.float32)
    h = backend.scene_create(sc)
    try:
        backend.scene_set_materials(h, prm, np.zeros(sc.n_tris, np.int32))
        g = torch.zeros(8, device="cuda")
        dl = torch.full((w * w * 3,), value, device="cuda")
        torch.cuda.synchronize()
        backend.backward(h, cam, cfg, 5, dl.data_ptr(), g.data_ptr())
        backend.sync()
    finally:
        backend.scene_destroy(h)
    want = float(np.float32(value) * np.float32(1 / spp)) * w * w * spp
    units = (256 * 2 + 14) / 2 + 148 / 2
    assert abs(float(g[4]) - want) <= units * 2.0 ** -24 * want
