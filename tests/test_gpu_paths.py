"""The plain path tracer's task loop (rm_paths.cu) at the sizes where it changes
form: one, 8 and 32 lanes per pixel, sample counts that leave a partial last
round, the adaptive test after some rounds (segments), frames of more and of
fewer lanes than one wave of resident blocks holds, several light candidates,
partially transparent scenes, no bounce at all, and more samples than one chunk
or one segment holds.  Radiance, RGB8 and sample counts equal the oracle's bit
for bit, the large ones the batch renderer's."""
import numpy as np
import pytest

from raymotion_b200 import BatchItem, RenderConfig, _abi
from raymotion_b200.scenes import PLAIN_FLAGS, cornell_box, sized_field

pytestmark = pytest.mark.gpu


def _cfg(w, h, spp, depth, adapt=None, candidates=1, flags=PLAIN_FLAGS):
    c = RenderConfig(width=w, height=h, spp=spp, max_bounces=depth, restir_candidates=candidates, restir_spatial=0,
                     flags=flags)
    c.adapt_min, c.adapt_step = adapt if adapt else (0, 8)
    if candidates > 1:
        c.flags &= ~_abi.RM_FLAG_RESTIR_OFF
    return c


CASES = {
    "one_lane": _cfg(97, 41, 5, 5),
    "one_lane_adaptive": _cfg(53, 31, 30, 4, adapt=(10, 5)),
    "eight_partial_round": _cfg(141, 71, 9, 4),
    "eight_segments": _cfg(143, 71, 27, 4, adapt=(8, 8)),
    "eight_segments_one_wave": _cfg(40, 21, 27, 4, adapt=(8, 8)),
    "thirty_two_partial_round": _cfg(67, 41, 70, 3),
    "thirty_two_segments": _cfg(66, 39, 96, 3, adapt=(32, 32)),
    "candidates": _cfg(141, 71, 8, 4, candidates=8),
    "candidates_segments": _cfg(141, 71, 24, 3, adapt=(8, 8), candidates=3),
    "no_bounce": _cfg(60, 33, 8, 0),
    "one_pixel": _cfg(1, 1, 64, 6),
}


@pytest.mark.parametrize("scene", ["cornell", "field", "transparent"])
@pytest.mark.parametrize("name", list(CASES))
def test_frames_equal_the_oracle(backend, oracle, name, scene):
    cfg = CASES[name]
    if scene == "field":
        sb, cam, _ = sized_field(5, 3000, cfg.width, cfg.height, cfg.spp, cfg.max_bounces)
    else:
        sb, cam, _ = cornell_box(2)
    sc = sb.pack()
    if scene == "transparent":
        sc.tris["alpha"][20:28] = 0.4
    sc = oracle.with_reference_bvh(sc)
    backend.stats_reset()
    rgb, hdr = backend.render(sc, cam, cfg, seed=77, hdr=True, use_nodes=False)
    st = backend.stats()
    o_rgb, o_hdr, o_st = oracle.Oracle().render(sc, cam, cfg, 77)
    assert np.array_equal(hdr.view(np.uint32), np.asarray(o_hdr).reshape(-1).view(np.uint32))
    assert np.array_equal(rgb, o_rgb)
    assert st["path_samples"] == o_st["path_samples"]


@pytest.mark.parametrize("w,h,spp,depth", [(160, 120, 1024, 2), (60, 41, 4200, 2)], ids=["two_chunks", "cut_segment"])
def test_large_sample_counts_equal_the_batch(backend, w, h, spp, depth):
    import torch
    sb, cam, _ = cornell_box(3)
    cfg = _cfg(w, h, spp, depth)
    scene = backend.scene_create(sb.pack())
    n = w * h * 3
    out = [(torch.empty(n, dtype=torch.uint8, device="cuda"), torch.empty(n, device="cuda")) for _ in range(2)]
    aux = torch.empty(w * h * 2, dtype=torch.int32, device="cuda")
    backend.render_scene_async(scene, cam, cfg, 9, out[0][0].data_ptr(), out[0][1].data_ptr())
    backend.sync()
    states = backend.debug_read(4, w * h)
    backend.render_batch([BatchItem(scene, cam, cfg, 9, out[1][0].data_ptr(), out[1][1].data_ptr(), aux.data_ptr())])
    assert torch.equal(out[0][0], out[1][0]) and torch.equal(out[0][1], out[1][1])
    assert np.array_equal(states, aux.cpu().numpy().view(np.uint32))
    backend.scene_destroy(scene)
