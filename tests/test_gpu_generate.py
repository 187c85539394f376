"""The two forms of the ReSTIR candidate pass: tiles of 8 x 4 pixels with their
visibility rays sorted by light (up to 4,096 pixels per SM), and a thread a
pixel.  At sizes around a tile, with candidate counts that do not divide among a
pixel's four threads, with one light and with many, and on the other side of the
line, the frames (undenoised) equal the oracle's bit for bit."""
import numpy as np
import pytest

from raymotion_b200 import RenderConfig, _abi
from raymotion_b200.scenes import cornell_box, sized_field

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scene", ["cornell", "field"])
@pytest.mark.parametrize("w,h,candidates", [(1, 1, 32), (8, 4, 2), (9, 5, 5), (7, 3, 1), (67, 33, 31), (130, 71, 32),
                                            (40, 24, 50), (1013, 600, 3)])
def test_frames_equal_the_oracle(backend, oracle, scene, w, h, candidates):
    cfg = RenderConfig(width=w, height=h, spp=1, max_bounces=2, restir_candidates=candidates, restir_spatial=2,
                       restir_radius=10.0, flags=_abi.RM_FLAG_NO_ENV | _abi.RM_FLAG_DENOISE_OFF)
    cfg.adapt_min = 0
    sb, cam = cornell_box(3)[:2] if scene == "cornell" else sized_field(9, 3000, w, h, 1, 2)[:2]
    sc = oracle.with_reference_bvh(sb.pack())
    backend.reset_history()
    rgb, hdr = backend.render(sc, cam, cfg, seed=31, hdr=True, use_nodes=False)
    assert backend.stats()["kernel_chain"] == 2
    o_rgb, o_hdr, _ = oracle.Oracle().render(sc, cam, cfg, 31)
    assert np.array_equal(hdr.view(np.uint32), np.asarray(o_hdr).reshape(-1).view(np.uint32))
    assert np.array_equal(rgb, o_rgb)
