"""Scene uploads at the sizes where their steps change form: the check of the
triangles (host up to 2,048, device above), a resident scene kept when an upload
is rejected, and the 4-wide collapse (rm_quad.cu: one block up to 2,048 binary
records, twelve launches and one block up to 65,536, a launch per level above)."""
import numpy as np
import pytest

from raymotion_b200 import RenderConfig, RenderError, _abi
from raymotion_b200.scene import Camera

from .gpu_util import random_rays
from .test_gpu_quads import _check, _soup, _trace

pytestmark = pytest.mark.gpu


def _variant(sc, **fields):
    tris = sc.tris.copy()
    for k, v in fields.items():
        tris[k][-1] = v
    return type(sc)(tris=tris, light_tri=sc.light_tri, light_cdf=sc.light_cdf, light_total=sc.light_total,
                    texels=sc.texels, verts64=sc.verts64)


@pytest.mark.parametrize("records", [2047, 2048, 2049, 65535, 65536, 65537])
def test_collapse_forms(backend, oracle, records, monkeypatch):
    monkeypatch.setenv("RAYMOTION_CUDA_BVH_LEAF", "1")
    sc = oracle.with_reference_bvh(_soup(records + 1, records, spread=12.0))
    backend.upload(sc, use_nodes=False)
    assert _check(backend, oracle, sc, random_rays(4000, [-13] * 3, [13] * 3, records)) > 0.0


@pytest.mark.parametrize("resident", [None, 2000, 5000])
@pytest.mark.parametrize("n", [1, 2048, 2049])
def test_rejected_upload_keeps_the_resident_scene(backend, n, resident):
    from raymotion_b200 import Backend
    b = Backend(0)
    rays = random_rays(2000, [-3] * 3, [3] * 3, 3)
    cfg = RenderConfig(width=16, height=9, spp=1, max_bounces=2, adapt_min=0, flags=_abi.RM_FLAG_NO_ENV)
    before = None
    if resident:
        b.upload(_soup(resident, 2), use_nodes=False)
        before = _trace(b, rays)
    good = _soup(n, 4)
    for bad in (dict(texture_offset=0), dict(texture_offset=0, texture_width=1, texture_height=1)):
        with pytest.raises(RenderError, match="texture outside") as e:
            b.upload(_variant(good, **bad), use_nodes=False)
        assert e.value.code == _abi.RM_ERR_INVALID
    if resident:
        assert all(np.array_equal(x, y) for x, y in zip(before, _trace(b, rays)))
    else:
        with pytest.raises(RenderError, match="no resident scene"):
            b.render_resident_async(Camera(), cfg, 1, None)
    b.upload(good, use_nodes=False)
    after = _trace(b, rays)
    b.upload(_variant(good), use_nodes=False)  # the same bytes again: the BVH is kept
    assert b.stats()["bvh_kept"] == 1
    assert all(np.array_equal(x, y) for x, y in zip(after, _trace(b, rays)))
    b.close()


@pytest.mark.parametrize("n", [2048, 2049])
def test_opacity_is_found(backend, oracle, n):
    """A transparent triangle among many rules the ReSTIR chain out (its frames are of opaque scenes)."""
    from raymotion_b200.scenes import sized_field
    sb, cam, _ = sized_field(7, 1000, 32, 18, 1, 3)
    sc = sb.pack()
    tris = np.concatenate([sc.tris, np.repeat(sc.tris[:1], n - sc.n_tris)])
    cfg = RenderConfig(width=32, height=18, spp=1, max_bounces=3, adapt_min=0, restir_candidates=4, restir_spatial=2,
                       flags=_abi.RM_FLAG_NO_ENV)
    for alpha, chain in ((1.0, 2), (0.5, 1), (1.0, 2)):
        tris["alpha"][n // 2] = alpha
        s = type(sc)(tris=tris.copy(), light_tri=sc.light_tri, light_cdf=sc.light_cdf, light_total=sc.light_total,
                     texels=sc.texels, verts64=np.concatenate([tris[k] for k in ("v0", "v1", "v2")], axis=1))
        backend.render(s, cam, cfg, 1, use_nodes=False)
        assert backend.stats()["kernel_chain"] == chain
