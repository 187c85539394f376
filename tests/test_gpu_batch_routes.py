"""Which kernels a batch's images go through: up to 32 images of fewer than
65,536 samples, and every larger one, through the plain frame's (on several
streams); more small ones through the wavefront pool.  Both equal the
single-image renders bit for bit, in a batch of either kind and in one of both."""
import numpy as np
import pytest

from raymotion_b200 import BatchItem, RenderConfig
from raymotion_b200.scenes import PLAIN_FLAGS, sized_field

pytestmark = pytest.mark.gpu

# one, 8 and 32 lanes, partial rounds, the adaptive test, no bounce
CONFIGS = [dict(w=37, h=11, spp=3), dict(w=24, h=13, spp=9), dict(w=19, h=9, spp=33),
           dict(w=23, h=17, spp=24, adapt_min=8), dict(w=9, h=5, spp=8, depth=0)]
LARGE = dict(w=257, h=128, spp=2)      # 65,792 samples
BELOW = dict(w=257, h=127, spp=2)      # 65,278


def _item(k, w, h, spp, depth=5, adapt_min=0):
    cfg = RenderConfig(width=w, height=h, spp=spp, max_bounces=depth, restir_candidates=1 + 3 * (k % 2),
                       restir_spatial=0, flags=PLAIN_FLAGS)
    cfg.adapt_min, cfg.adapt_step = adapt_min, 8
    return cfg


@pytest.mark.parametrize("name,specs,pool", [
    ("few_small", [CONFIGS[k % 5] for k in range(32)], False),
    ("many_small", [CONFIGS[k % 5] for k in range(33)], True),
    ("both", [CONFIGS[k % 5] for k in range(32)] + [LARGE, BELOW, LARGE], True),
    ("one_large", [LARGE], False),
])
@pytest.mark.parametrize("tuning", [{}, dict(pool_chunks=7, tile_shape=1, grid_scale=1, graph_waves=2, bvh_width=8)],
                         ids=["default", "tiny_pool_wide"])
def test_batches_equal_single_images(backend, name, specs, pool, tuning):
    import torch
    scenes = []
    for seed, alpha in ((5, 1.0), (6, 0.5)):
        sb, cam, _ = sized_field(seed, 1500, 64, 36, 1, 4)
        sc = sb.pack()
        if alpha < 1.0:
            sc.tris["alpha"][::7] = alpha
        scenes.append((backend.scene_create(sc), cam))
    default = backend.batch_tuning()
    try:
        items, outs, want = [], [], []
        for k, spec in enumerate(specs):
            h, cam = scenes[(k // 5) % 2]
            cfg = _item(k, **spec)
            n = cfg.width * cfg.height
            ref = torch.empty(n * 3, device="cuda")
            backend.render_scene_async(h, cam, cfg, 40 + k, None, ref.data_ptr())
            backend.sync()
            want.append((ref, backend.debug_read(4, n)))
            # outputs a caller does not want are left out
            o = dict(hdr=torch.full((n * 3,), -1.0, device="cuda"),
                     rgb=torch.full((n * 3,), 7, dtype=torch.uint8, device="cuda") if k % 3 else None,
                     aux=torch.zeros(n * 2, dtype=torch.int32, device="cuda") if k % 2 else None)
            outs.append(o)
            items.append(BatchItem(h, cam, cfg, 40 + k, *(None if o[x] is None else o[x].data_ptr()
                                                          for x in ("rgb", "hdr", "aux"))))
        if tuning:
            backend.set_batch_tuning(**tuning)
        backend.render_batch(items)
        assert (len(backend.batch_log()) > 0) == pool
        for o, (ref, aux) in zip(outs, want):
            assert torch.equal(o["hdr"].view(torch.int32), ref.view(torch.int32))
            if o["aux"] is not None:
                assert np.array_equal(o["aux"].cpu().numpy().view(np.uint32), aux)
            assert o["rgb"] is None or int((o["rgb"] != 7).sum()) > 0
    finally:
        backend.set_batch_tuning(**default)
        for h, _ in scenes:
            backend.scene_destroy(h)
