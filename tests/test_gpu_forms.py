"""The forms of the renderers that a default call of a test's size does not take.

Frames of up to two waves of resident tail blocks (151,552 pixels on 148 SMs) are
all tail unless RAYMOTION_CUDA_TAIL is set, and batches of up to 32 small images
bypass the path-slot pool, so these tests set the hand-over and fill the pool,
and look at the logs of both to see that they ran.  The plain path's chunks and
cut segments are compared with the oracle, which has neither."""
import numpy as np
import pytest

from raymotion_b200 import BatchItem, RenderConfig, _abi
from raymotion_b200.scenes import cornell_box, icosphere_field, sized_field

from .gpu_util import exact_fraction
from .test_gpu_batch import TUNINGS, _cfg, _mixed_images
from .test_gpu_paths import _cfg as _plain

pytestmark = pytest.mark.gpu

WAVES = {
    "merged": {},
    "wide": dict(RAYMOTION_CUDA_WIDE="1"),
    "split": dict(RAYMOTION_CUDA_SPLIT_WAVES="1"),
    "split_wide": dict(RAYMOTION_CUDA_SPLIT_WAVES="1", RAYMOTION_CUDA_WIDE="1"),
    "one_stream": dict(RAYMOTION_CUDA_STREAMS="1"),
    "four_streams": dict(RAYMOTION_CUDA_STREAMS="4"),
    "count_wait": dict(RAYMOTION_CUDA_COUNT_LAG="0"),
}
HAND_OVER = ["0", "4000"]  # unfinished paths: never, and in the middle of the frame with shadow rays pending


def _waves(backend, oracle, sc, cam, cfg, seeds, tail):
    o = oracle.Oracle()
    backend.reset_history()
    npix = cfg.width * cfg.height
    for seed in seeds:
        _, o_hdr, o_st = o.render(sc, cam, cfg, seed)
        _, g_hdr = backend.render(sc, cam, cfg, seed, hdr=True)
        assert o_st["chain"] == 2 and backend.stats()["kernel_chain"] == 2
        assert np.array_equal(backend.debug_read(4, npix), o.debug_read(4, npix))
        assert exact_fraction(g_hdr, o_hdr) == 1.0
        log = backend.wave_log()
        assert len(log) > 2 and log[0, 0] > tail and not log[-1, :3].any()
    return log


@pytest.mark.parametrize("tail", HAND_OVER)
@pytest.mark.parametrize("form", list(WAVES))
def test_waves_match_the_oracle(backend, oracle, form, tail, monkeypatch):
    for k, v in WAVES[form].items():
        monkeypatch.setenv(k, v)
    monkeypatch.setenv("RAYMOTION_CUDA_TAIL", tail)
    sb, cam, _ = sized_field(4, 4000, 160, 90, 4, 6)
    sc = oracle.with_reference_bvh(sb.pack())
    cfg = RenderConfig(width=160, height=90, spp=4, max_bounces=6, adapt_min=0, restir_candidates=8, restir_spatial=4,
                       restir_radius=12.0, flags=_abi.RM_FLAG_NO_ENV | _abi.RM_FLAG_DENOISE_OFF)
    # the second frame reuses the first as temporal history
    log = _waves(backend, oracle, sc, cam, cfg, (11, 12), int(tail))
    assert (log[:-1, 2] > 0).any()  # (shadow rays were queued)


@pytest.mark.parametrize("split", [False, True], ids=["merged", "split"])
@pytest.mark.parametrize("candidates,flags", [(1, 0), (8, _abi.RM_FLAG_NOMIS), (4, _abi.RM_FLAG_NO_RR)])
def test_wave_shading_matches_the_oracle(backend, oracle, candidates, flags, split, monkeypatch):
    monkeypatch.setenv("RAYMOTION_CUDA_TAIL", "0")
    if split:
        monkeypatch.setenv("RAYMOTION_CUDA_SPLIT_WAVES", "1")
    sb, cam, _ = icosphere_field(seed=7, n_spheres=24, subdiv=2, n_emitters=48, width=96, height=64, spp=6, depth=7)
    sc = oracle.with_reference_bvh(sb.pack())
    cfg = RenderConfig(width=96, height=64, spp=6, max_bounces=7, adapt_min=0, restir_candidates=candidates,
                       restir_spatial=3, restir_radius=9.0, flags=_abi.RM_FLAG_NO_ENV | _abi.RM_FLAG_DENOISE_OFF | flags)
    _waves(backend, oracle, sc, cam, cfg, (99,), 0)


@pytest.mark.parametrize("parts,height", [(4, 3), (4, 4), (3, 7), (2, 1)])
def test_waves_of_few_rows(backend, oracle, parts, height, monkeypatch):
    monkeypatch.setenv("RAYMOTION_CUDA_TAIL", "0")
    monkeypatch.setenv("RAYMOTION_CUDA_STREAMS", str(parts))
    sb, cam, _ = sized_field(4, 4000, 96, height, 4, 6)
    sc = oracle.with_reference_bvh(sb.pack())
    cfg = RenderConfig(width=96, height=height, spp=4, max_bounces=6, adapt_min=0, restir_candidates=8,
                       restir_spatial=4, restir_radius=12.0, flags=_abi.RM_FLAG_NO_ENV | _abi.RM_FLAG_DENOISE_OFF)
    _waves(backend, oracle, sc, cam, cfg, (31,), 0)


@pytest.mark.parametrize("tuning", TUNINGS, ids=["default", "tiny_pool_graph2", "small_pool_nograph", "wide_bvh"])
def test_pool_tunings_equal_single_images(backend, tuning):
    """35 images of fewer than 65,536 samples each, in every shape of the batch tests."""
    import torch
    images = [(sc, cam, cfg, seed) for sc, cam, cfg, seed, _ in _mixed_images()]
    small = [x for x in images if x[2].width * x[2].height * x[2].spp < 65536]
    big = [(sc, cam, _cfg(cfg, width=cfg.width // 3, height=cfg.height // 3), seed)
           for sc, cam, cfg, seed in images if cfg.width * cfg.height * cfg.spp >= 65536]
    images = small + big
    images = [(*images[k % len(images)][:3], 500 + k) for k in range(35)]
    assert all(c.width * c.height * c.spp < 65536 for _, _, c, _ in images)
    handles, items, outs, refs = {}, [], [], []
    try:
        for sc, cam, cfg, seed in images:
            if id(sc) not in handles:
                handles[id(sc)] = backend.scene_create(sc)
            n = cfg.width * cfg.height
            pair = [torch.full((n * 3,), -1.0, device="cuda") for _ in range(2)]
            aux = torch.zeros(n * 2, dtype=torch.int32, device="cuda")
            backend.render_scene_async(handles[id(sc)], cam, cfg, seed, None, pair[0].data_ptr())
            backend.sync()
            refs.append((pair[0], backend.debug_read(4, n)))
            outs.append((pair[1], aux))
            items.append(BatchItem(handles[id(sc)], cam, cfg, seed, None, pair[1].data_ptr(), aux.data_ptr()))
        backend.set_batch_tuning(**tuning)
        backend.render_batch(items)
        assert len(backend.batch_log()) > 0  # through the pool
    finally:
        backend.set_batch_tuning(**TUNINGS[0])
        for h in handles.values():
            backend.scene_destroy(h)
    assert backend.stats()["device_error"] == 0
    for k, ((hdr, aux), (ref, dbg)) in enumerate(zip(outs, refs)):
        assert torch.equal(hdr.view(torch.int32), ref.view(torch.int32)), k
        assert np.array_equal(aux.cpu().numpy().view(np.uint32), dbg), k


@pytest.mark.parametrize("w,h,spp", [(160, 120, 1024), (60, 41, 4200)], ids=["two_chunks", "cut_segment"])
def test_large_sample_counts_equal_the_oracle(backend, oracle, w, h, spp):
    sb, cam, _ = cornell_box(3)
    sc = oracle.with_reference_bvh(sb.pack())
    cfg = _plain(w, h, spp, 2)
    rgb, hdr = backend.render(sc, cam, cfg, seed=9, hdr=True, use_nodes=False)
    o = oracle.Oracle()
    o_rgb, o_hdr, _ = o.render(sc, cam, cfg, 9)
    assert np.array_equal(hdr.view(np.uint32), np.asarray(o_hdr).reshape(-1).view(np.uint32))
    assert np.array_equal(rgb, o_rgb)
    assert np.array_equal(backend.debug_read(4, w * h), o.debug_read(4, w * h))


def test_frames_whose_pixels_stop_early(backend, oracle):
    """Frames of many segments whose adaptive test soon stops every pixel, the
    rest of whose launches the host may save, between frames that go on, alone and
    in a batch on several streams: all equal the oracle."""
    import torch

    from . import kat_scenes as K
    even = oracle.with_reference_bvh(K.fullscreen_emitter())
    noisy = oracle.with_reference_bvh(cornell_box(3)[0].pack())
    cam = cornell_box(3)[1]
    cfgs = {id(even): _plain(160, 90, 512, 2, adapt=(16, 8)), id(noisy): _plain(40, 30, 96, 3, adapt=(16, 8))}
    for c in cfgs.values():
        c.adapt_rel, c.adapt_abs = 0.02, 0.002
    order = [even, noisy, even, even, noisy, noisy, even, noisy]
    want = {id(s): oracle.Oracle().render(s, cam, cfgs[id(s)], 5)[1].reshape(-1) for s in (even, noisy)}
    handles = {id(s): backend.scene_create(s) for s in (even, noisy)}
    try:
        outs = [torch.empty(cfgs[id(s)].width * cfgs[id(s)].height * 3, device="cuda") for s in order]
        for s, o in zip(order, outs):  # one after the other, not waited for
            backend.render_scene_async(handles[id(s)], cam, cfgs[id(s)], 5, None, o.data_ptr())
        backend.sync()
        alone = [o.cpu().numpy() for o in outs]
        for o in outs:
            o.zero_()
        backend.render_batch([BatchItem(handles[id(s)], cam, cfgs[id(s)], 5, None, o.data_ptr(), None)
                              for s, o in zip(order, outs)])
        for s, a, o in zip(order, alone, outs):
            ref = np.asarray(want[id(s)], np.float32)
            assert np.array_equal(a.view(np.uint32), ref.view(np.uint32))
            assert np.array_equal(o.cpu().numpy().view(np.uint32), ref.view(np.uint32))
    finally:
        for h in handles.values():
            backend.scene_destroy(h)
