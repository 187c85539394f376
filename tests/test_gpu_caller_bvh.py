"""Caller BVHs whose shape the collapses (rm_quad.cu, rm_wide.cu) cannot take as
they take a built one: subtrees that several nodes share, leaves that overlap,
boxes that do not hold their children's or have their bounds swapped.  Hits equal the oracle's
bit for bit (they do not depend on the BVH); any-hit agrees."""
import numpy as np
import pytest

from raymotion_b200 import RenderError, _abi

from .gpu_util import random_rays
from .test_gpu_quads import _check, _soup, _trace

pytestmark = pytest.mark.gpu


class Node:
    """An inner node of two children, each a Node or a list of triangles; a
    Node or list given to several parents is one node of the array."""

    def __init__(self, left, right):
        self.left, self.right = left, right


def caller_bvh(sc, root, box=None):
    """sc with the BVH of `root` as the caller's own: parents before their
    children.  box(object, depth, mn, mx) may change a node's box."""
    order, place = [], {}
    todo = [(root, 1)]
    depth = {}
    while todo:  # a node's place: behind all of its parents'
        t, d = todo.pop()
        if depth.get(id(t), 0) >= d:
            continue
        depth[id(t)] = d
        place[id(t)] = t
        if isinstance(t, Node):
            todo += [(t.left, d + 1), (t.right, d + 1)]
    objects = sorted(place.values(), key=lambda t: depth[id(t)])
    index = {id(t): i for i, t in enumerate(objects)}
    bounds = {}
    for t in reversed(objects):
        if isinstance(t, Node):
            a, b = bounds[id(t.left)], bounds[id(t.right)]
            bounds[id(t)] = (np.minimum(a[0], b[0]), np.maximum(a[1], b[1]))
        else:
            v = np.concatenate([sc.tris[k][t] for k in ("v0", "v1", "v2")])
            bounds[id(t)] = (v.min(0), v.max(0))
    arr = np.zeros(len(objects), _abi.BVH_NODE_DTYPE)
    for i, t in enumerate(objects):
        mn, mx = bounds[id(t)]
        if box:
            mn, mx = box(t, depth[id(t)], mn, mx)
        if isinstance(t, Node):
            arr[i] = (tuple(mn), tuple(mx), index[id(t.left)], index[id(t.right)], 0, 0)
        else:
            arr[i] = (tuple(mn), tuple(mx), -1, -1, len(order), len(t))
            order += t
    assert sorted(order) == list(range(sc.n_tris))
    return type(sc)(tris=sc.tris, light_tri=sc.light_tri, light_cdf=sc.light_cdf, light_total=sc.light_total,
                    texels=sc.texels, verts64=sc.verts64, nodes=arr, bvh_tri=np.asarray(order, np.int32))


def _twice(levels):
    """A chain that names its next level as both children."""
    t = Node([0], [1, 2])
    for _ in range(levels):
        t = Node(t, t)
    return t


def _two_parents():
    a = Node([2], Node([3, 4], [5]))
    return Node(Node([0], a), Node(Node([1], a), [6]))


SHARED = {"child_twice": (3, lambda: _twice(1)), "chain": (3, lambda: _twice(8)), "two_parents": (7, _two_parents),
          "shared_leaf": (2, lambda: (lambda a: Node(Node(a, [1]), a))([0]))}


@pytest.mark.parametrize("wide", [False, True], ids=["default", "wide"])
@pytest.mark.parametrize("shape", list(SHARED))
def test_shared_subtrees(backend, oracle, shape, wide, monkeypatch):
    if wide:
        monkeypatch.setenv("RAYMOTION_CUDA_WIDE", "1")
    n, root = SHARED[shape]
    sc = oracle.with_reference_bvh(_soup(n, 31, spread=1.0))
    backend.upload(caller_bvh(sc, root()), use_nodes=True)
    rays = random_rays(4000, [-2, -2, -2], [2, 2, 2], n)
    assert _check(backend, oracle, sc, rays) > 0.0


def test_shared_subtrees_are_bounded(backend, oracle):
    """Two to the 30 paths: refused on the host like any BVH of too many nodes."""
    sc = oracle.with_reference_bvh(_soup(3, 31))
    with pytest.raises(RenderError, match="shared subtrees") as e:
        backend.upload(caller_bvh(sc, _twice(30)), use_nodes=True)
    assert e.value.code == _abi.RM_ERR_BVH


def test_overlapping_leaves_in_the_wide_bvh(backend, oracle, monkeypatch):
    """Two leaves over one range of triangles: more triangles in leaves than the scene has."""
    monkeypatch.setenv("RAYMOTION_CUDA_WIDE", "1")
    sc = oracle.with_reference_bvh(_soup(8, 32, spread=1.0))
    caller = caller_bvh(sc, Node(Node([0, 1, 2], [3, 4]), Node([5], [6, 7])))
    leaf = [i for i in range(len(caller.nodes)) if caller.nodes["count"][i] > 0]
    for i in leaf:  # every leaf: the first four positions, or the last four
        caller.nodes[i]["count"], caller.nodes[i]["offset"] = 4, 0 if i in leaf[:2] else 4
        caller.nodes[i]["mn"], caller.nodes[i]["mx"] = caller.nodes[0]["mn"], caller.nodes[0]["mx"]
    for i in set(range(len(caller.nodes))) - set(leaf):
        caller.nodes[i]["mn"], caller.nodes[i]["mx"] = caller.nodes[0]["mn"], caller.nodes[0]["mx"]
    backend.upload(caller, use_nodes=True)
    rays = random_rays(4000, [-2, -2, -2], [2, 2, 2], 8)
    assert _check(backend, oracle, sc, rays) > 0.0


def test_most_subtrees_pending(backend, oracle):
    """64 levels whose every node holds the rest of the chain and a larger subtree
    of three leaves: the collapse opens that subtree twice, so that each 4-wide
    node pushes three subtrees and the chain goes on one level further down.  All
    boxes hold the rays' origins and the chain is entered first."""
    inner = 62  # (the leaves of the last subtree are on level 64)
    n = 3 * (inner - 1) + 2
    sc = oracle.with_reference_bvh(_soup(n, 33, spread=1.0))
    tri = iter(range(n))
    rest, size, half = Node([next(tri)], [next(tri)]), {}, 4.0
    size[id(rest)] = half
    for _ in range(inner - 1):
        half /= 0.98
        pair = Node([next(tri)], [next(tri)])
        three = Node([next(tri)], pair)
        rest = Node(rest, three)
        size.update({id(pair): 0.99 * half, id(three): half, id(rest): half})
    assert next(tri, None) is None

    def box(t, depth, mn, mx):
        h = size.get(id(t), 3.9)  # (a leaf holds the origins too)
        assert (mn > -h).all() and (mx < h).all()
        return np.full(3, -h, np.float32), np.full(3, h, np.float32)

    builds = backend.stats()["bvh_builds"]
    backend.upload(caller_bvh(sc, rest, box), use_nodes=True)
    assert backend.stats()["bvh_builds"] == builds  # not too deep for the caller's BVH
    rays = random_rays(4000, [-1.5] * 3, [1.5] * 3, 34)
    assert _check(backend, oracle, sc, rays) > 0.05


@pytest.mark.parametrize("wide", [False, True], ids=["default", "wide"])
@pytest.mark.parametrize("what", ["too_small", "swapped_inner", "swapped_leaf", "swapped_one_axis"])
def test_boxes_are_taken_as_given(backend, oracle, what, wide, monkeypatch):
    """A subtree is entered through every box on its way, as the reference enters
    it, also where an inner box misses part of it or gives its bounds the other
    way round; the oracle walks the same nodes."""
    if wide:
        monkeypatch.setenv("RAYMOTION_CUDA_WIDE", "1")
    sc = oracle.with_reference_bvh(_soup(200, 35))
    nodes = sc.nodes.copy()
    inner = nodes["count"] == 0
    pick = {"too_small": inner, "swapped_inner": inner}.get(what, ~inner)
    pick = np.flatnonzero(pick)[1::3]
    mn, mx = nodes["mn"].copy(), nodes["mx"].copy()
    if what == "too_small":
        nodes["mn"][pick], nodes["mx"][pick] = mn[pick] + 0.3 * (mx - mn)[pick], mx[pick] - 0.3 * (mx - mn)[pick]
    else:
        axes = [1] if what == "swapped_one_axis" else [0, 1, 2]
        for a in axes:
            nodes["mn"][pick, a], nodes["mx"][pick, a] = mx[pick, a], mn[pick, a]
    caller = type(sc)(tris=sc.tris, light_tri=sc.light_tri, light_cdf=sc.light_cdf, light_total=sc.light_total,
                      texels=sc.texels, verts64=sc.verts64, nodes=nodes, bvh_tri=sc.bvh_tri)
    backend.upload(caller, use_nodes=True)
    rays = random_rays(8000, [-3, -3, -3], [3, 3, 3], 36)
    every = (oracle.trace(sc, rays)[0] >= 0).mean()
    if what == "too_small":
        # (which hit is the closest of those found depends on the order of the visits)
        hit = oracle.trace(caller, rays, any_hit=True)[0] >= 0
        assert np.array_equal(_trace(backend, rays, any_hit=True)[0] >= 0, hit)
        assert 0 < hit.mean() < every
    else:
        assert _check(backend, oracle, caller, rays) == every


@pytest.mark.parametrize("shape", list(SHARED))
def test_update_of_shared_subtrees(backend, oracle, shape):
    """A subtree with several parents has no one place to pass its new box on to."""
    n, root = SHARED[shape]
    sc = oracle.with_reference_bvh(_soup(n, 31, spread=1.0))
    backend.upload(caller_bvh(sc, root()), use_nodes=True)
    moved = sc.tris.copy()
    for f in ("v0", "v1", "v2"):
        moved[f] += np.float32(3.0)
    backend.update(moved, rebuild_every=0)
    v64 = np.concatenate([moved["v0"], moved["v1"], moved["v2"]], axis=1).astype(np.float64)
    ms = oracle.with_reference_bvh(type(sc)(tris=moved, light_tri=sc.light_tri, light_cdf=sc.light_cdf,
                                            light_total=sc.light_total, texels=sc.texels, verts64=v64))
    assert _check(backend, oracle, ms, random_rays(4000, [1, 1, 1], [5, 5, 5], n)) > 0.0
