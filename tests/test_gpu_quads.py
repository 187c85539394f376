"""The 4-wide BVH (rm_quad.cu) where its collapse can go wrong: trees of a few
triangles, leaves of one, two and many triangles, and a chain as deep as the
binary tree may be (its collapse keeps the most subtrees pending).  Hits equal
the oracle's bit for bit (they do not depend on the BVH); any-hit agrees."""
import numpy as np
import pytest

from raymotion_b200 import _abi
from raymotion_b200.scene import SceneBuilder

from .gpu_util import random_rays

pytestmark = pytest.mark.gpu


def _trace(backend, rays, any_hit=False):
    import torch
    n = len(rays)
    d = torch.from_numpy(rays).cuda()
    tri = torch.empty(n, dtype=torch.int32, device="cuda")
    t, u, v = (torch.empty(n, device="cuda") for _ in range(3))
    backend.trace(d.data_ptr(), n, any_hit, tri.data_ptr(), t.data_ptr(), u.data_ptr(), v.data_ptr())
    return [x.cpu().numpy() for x in (tri, t, u, v)]


def _soup(n, seed, spread=2.0):
    rng = np.random.default_rng(seed)
    sb = SceneBuilder()
    c = rng.uniform(-spread, spread, (n, 3))
    sb.add_triangles(c, c + rng.normal(0, 0.6, (n, 3)), c + rng.normal(0, 0.6, (n, 3)))
    return sb.pack()


def _check(backend, oracle, sc, rays):
    g = _trace(backend, rays)
    ref = oracle.trace(sc, rays)
    assert np.array_equal(g[0], ref[0])
    hit = ref[0] >= 0
    for a, b in zip(g[1:], ref[1:]):
        assert np.array_equal(a[hit].view(np.uint32), b[hit].view(np.uint32))
    assert np.array_equal(_trace(backend, rays, any_hit=True)[0] >= 0, hit)
    return hit.mean()


@pytest.mark.parametrize("leaf", ["1", "2", "255"])
@pytest.mark.parametrize("n", [1, 2, 3, 4, 5, 6, 9, 17, 63, 257, 1000])
def test_small_trees_and_leaf_sizes(backend, oracle, n, leaf, monkeypatch):
    monkeypatch.setenv("RAYMOTION_CUDA_BVH_LEAF", leaf)
    sc = oracle.with_reference_bvh(_soup(n, n))
    rays = random_rays(4000, [-3, -3, -3], [3, 3, 3], n)
    backend.upload(sc, use_nodes=False)
    assert _check(backend, oracle, sc, rays) > 0.0
    moved = sc.tris.copy()
    for f in ("v0", "v1", "v2"):
        moved[f] += np.float32(0.25)
    backend.update(moved, rebuild_every=0)  # the refit's copy into the 4-wide nodes
    v64 = np.concatenate([moved["v0"], moved["v1"], moved["v2"]], axis=1).astype(np.float64)
    ms = oracle.with_reference_bvh(type(sc)(tris=moved, light_tri=sc.light_tri, light_cdf=sc.light_cdf,
                                            light_total=sc.light_total, texels=sc.texels, verts64=v64))
    _check(backend, oracle, ms, rays)


@pytest.mark.parametrize("shape", ["chain", "bushy_chain"])
def test_deepest_caller_bvh(backend, oracle, shape):
    """64 levels: a chain of leaves, and one whose every second level holds a
    subtree of two leaves (three subtrees pending per two levels)."""
    depth = 63  # internal nodes on the chain: the last leaf is on level 64
    paired = {k for k in range(depth - 1) if k % 2} if shape == "bushy_chain" else set()
    n = depth + 1 + len(paired)
    sc = oracle.with_reference_bvh(_soup(n, 5))
    tri = iter(range(n))
    tree = next(tri)
    for level in reversed(range(depth)):
        tree = ((next(tri), next(tri)) if level in paired else next(tri), tree)
    assert next(tri, None) is None

    def leaves(t):
        return [t] if not isinstance(t, tuple) else leaves(t[0]) + leaves(t[1])

    order = []
    nodes = []

    def emit(t):
        i = len(nodes)
        nodes.append(None)
        ids = leaves(t)
        v = np.concatenate([sc.tris[k][ids] for k in ("v0", "v1", "v2")])
        if not isinstance(t, tuple):
            nodes[i] = (v.min(0), v.max(0), -1, -1, len(order), 1)
            order.append(t)
        else:
            left = emit(t[0])
            right = emit(t[1])
            nodes[i] = (v.min(0), v.max(0), left, right, 0, 0)
        return i

    emit(tree)
    arr = np.zeros(len(nodes), _abi.BVH_NODE_DTYPE)
    for k, (mn, mx, left, right, off, cnt) in enumerate(nodes):
        arr[k] = (tuple(mn), tuple(mx), left, right, off, cnt)
    caller = type(sc)(tris=sc.tris, light_tri=sc.light_tri, light_cdf=sc.light_cdf, light_total=sc.light_total,
                      texels=sc.texels, verts64=sc.verts64, nodes=arr, bvh_tri=np.asarray(order, np.int32))
    backend.upload(caller, use_nodes=True)
    rays = random_rays(20000, [-3, -3, -3], [3, 3, 3], 9)
    assert _check(backend, oracle, sc, rays) > 0.05
