"""The build kernels at the sizes where they change form: the one-block LBVH of
the no-allocation query (powers of two of its sort, one triangle either side of
its limit, a triangle array that is not 16-byte aligned), and the clustering's
rounds around their tile (256) and around the count below which one block
finishes (2048).  Hits equal the oracle's bit for bit."""
import ctypes as C

import numpy as np
import pytest

from raymotion_b200 import _abi
from raymotion_b200.scene import SceneBuilder

from .gpu_util import random_rays

pytestmark = pytest.mark.gpu


def _soup(n, seed, clones=0):
    """n triangles, the last `clones` of them copies of one (equal codes, equal areas)."""
    rng = np.random.default_rng(seed)
    c = rng.uniform(-2, 2, (n, 3))
    a, b = c + rng.normal(0, 0.3, (n, 3)), c + rng.normal(0, 0.3, (n, 3))
    if clones:
        for v in (c, a, b):
            v[n - clones:] = v[n - clones]
    sb = SceneBuilder()
    sb.add_triangles(c, a, b)
    return sb.pack()


def _equal(got, ref, any_hit):
    if any_hit:
        assert np.array_equal(got[0] >= 0, ref[0] >= 0)
        return
    assert np.array_equal(got[0], ref[0])
    hit = ref[0] >= 0
    for a, b in zip(got[1:], ref[1:]):
        assert np.array_equal(a[hit].view(np.uint32), b[hit].view(np.uint32))


@pytest.mark.parametrize("offset", [0, 4], ids=["aligned", "unaligned"])
@pytest.mark.parametrize("n,clones", [(5, 0), (31, 0), (32, 0), (33, 0), (63, 60), (1024, 0), (1025, 700), (2047, 0),
                                      (2048, 0), (2048, 2048), (2049, 0), (4097, 0)])
def test_one_block_lbvh(backend, oracle, n, clones, offset):
    import torch
    sc = oracle.with_reference_bvh(_soup(n, n, clones))
    rays = random_rays(3000, [-3, -3, -3], [3, 3, 3], n)
    raw = torch.zeros(sc.n_tris * 176 + 16, dtype=torch.uint8, device="cuda")
    raw[offset:offset + sc.n_tris * 176] = torch.from_numpy(sc.tris.view(np.uint8).copy()).cuda()
    d = torch.from_numpy(rays).cuda()
    tri = torch.empty(len(rays), dtype=torch.int32, device="cuda")
    tuv = [torch.empty(len(rays), device="cuda") for _ in range(3)]
    err = C.create_string_buffer(512)
    for any_hit in (0, 1):
        rc = _abi.load_library().rmcuda_trace_noalloc(raw.data_ptr() + offset, sc.n_tris, d.data_ptr(), len(rays),
                                                      any_hit, tri.data_ptr(), *(x.data_ptr() for x in tuv), None, err,
                                                      512)
        assert rc == _abi.RM_OK, err.value
        _equal([x.cpu().numpy() for x in (tri, *tuv)], oracle.trace(sc, rays, any_hit=bool(any_hit)), any_hit)


@pytest.mark.parametrize("n,clones", [(255, 0), (257, 0), (2047, 0), (2048, 0), (2049, 0), (2049, 300), (2304, 0),
                                      (5000, 0), (6000, 2500), (40001, 0)])
def test_clustering_rounds(backend, oracle, n, clones):
    import torch
    sc = oracle.with_reference_bvh(_soup(n, n + 1, clones))
    rays = random_rays(6000, [-3, -3, -3], [3, 3, 3], n)
    backend.upload(sc, use_nodes=False)
    d = torch.from_numpy(rays).cuda()
    tri = torch.empty(len(rays), dtype=torch.int32, device="cuda")
    tuv = [torch.empty(len(rays), device="cuda") for _ in range(3)]
    for any_hit in (False, True):
        backend.trace(d.data_ptr(), len(rays), any_hit, tri.data_ptr(), *(x.data_ptr() for x in tuv))
        _equal([x.cpu().numpy() for x in (tri, *tuv)], oracle.trace(sc, rays, any_hit=any_hit), any_hit)
