"""The adjoint's task loop where it changes form: 32 lanes a pixel with a partial
last round, paths longer than the kept list (two walks a sample), samples with
clamped channels (the second walk takes their terms back out), partially
transparent scenes with one and with several light candidates, and more
materials than the block's sums hold.  Checked as in test_gpu_adjoint: FP64 central differences of the frozen-path renderer, the
same bounds (1e-3 of a gradient above 1 % of its kind's largest, else 1e-5 of
that largest), at a step of 1e-5: the renderer is double, and over long paths
inside glass the frame's third derivative in the index of refraction is too
large for 1e-3 (26 bounces, one material: 9.30e-4 there, 6.74e-4 at 1e-5)."""
import numpy as np
import pytest

from raymotion_b200 import _abi
from raymotion_b200.scenes import inverse_scene

from .test_gpu_adjoint import _grad, _set, _torch, central_difference

pytestmark = pytest.mark.gpu


def _case(oracle, spp=4, depth=6, w=40, h=33, alpha=None, candidates=1):
    d = inverse_scene(seed=7, n_spheres=10, subdiv=2, ground=20, patches=(3, 3), n_emitters=3, n_dielectric=8,
                      width=w, height=h, spp=spp, depth=depth)
    c = d["config"]
    c.restir_candidates, c.restir_spatial = candidates, 0
    if candidates > 1:
        c.flags &= ~_abi.RM_FLAG_RESTIR_OFF
    if alpha is not None:
        d["scene"].tris["alpha"][d["tri_material"] == 1] = alpha
        d["scene"].tris["alpha"][d["tri_material"] == 14] = alpha
    oracle.with_reference_bvh(d["scene"])
    return d


CASES = {
    "thirty_two_lanes": dict(spp=40),
    "two_walks": dict(depth=26),
    "transparent": dict(alpha=0.5),
    "transparent_ris": dict(alpha=0.5, candidates=4),
}


@pytest.mark.parametrize("name", list(CASES))
def test_adjoint_forms_match_fp64_central_differences(backend, oracle, name):
    torch = _torch()
    d = _case(oracle, **CASES[name])
    seed = 2024
    sc, cam, cfg, tm = d["scene"], d["camera"], d["config"], d["tri_material"]
    prm = d["params"].astype(np.float64)
    i64 = oracle.render_frozen(sc, cam, cfg, seed, tm, prm)
    T = i64 * 0.75 + 0.01
    dl = torch.from_numpy(((2.0 / i64.size) * (i64 - T)).astype(np.float32).ravel()).cuda()
    h = backend.scene_create(sc)
    try:
        _set(backend, h, d, d["params"])
        g = _grad(backend, h, d, seed, dl)
    finally:
        backend.scene_destroy(h)

    def loss(q):
        return np.mean((oracle.render_frozen(sc, cam, cfg, seed, tm, q) - T) ** 2)

    for col in (0, 3, 4, 7):
        cand = np.nonzero(d["mask"][:, col])[0]
        top = cand[np.argsort(-np.abs(g[cand, col]))][:2]
        fd = [central_difference(loss, prm, m, col, 1e-5) for m in top]
        big = max(abs(f) for f in fd)
        for m, f in zip(top, fd):
            tol = 1e-3 * abs(f) if abs(f) >= 1e-2 * big else 1e-5 * big
            assert abs(float(g[m, col]) - f) <= tol, f"material {m} param {col}: adjoint {g[m, col]} vs FD {f}"


@pytest.mark.parametrize("depth,w,h", [(6, 40, 33), (26, 40, 33), (6, 5, 3)])
def test_clamped_channels_take_no_gradient(backend, oracle, depth, w, h):
    """One sample a pixel: the clamped frame's gradient is the unclamped one's
    with dL/dI zero where the sample reaches the clamp.  The two differ by the
    order of at most 20 additions a sample and parameter, some added and taken
    out again: 2^-24 of the column's largest each."""
    torch = _torch()
    d = _case(oracle, spp=1, depth=depth, w=w, h=h)
    cfg = d["config"]
    hd = backend.scene_create(d["scene"])
    try:
        _set(backend, hd, d, d["params"])
        img = torch.empty(w * h * 3, dtype=torch.float32, device="cuda")
        backend.render_scene_async(hd, d["camera"], cfg, 3, None, img.data_ptr())
        backend.sync()
        clamp = 0.3 * float(img.max())
        dl = torch.linspace(0.1, 1.0, w * h * 3, device="cuda")
        whole = _grad(backend, hd, d, 3, dl)
        want = _grad(backend, hd, d, 3, torch.where(img < clamp, dl, 0.0).contiguous())
        cfg.clamp = clamp
        got = _grad(backend, hd, d, 3, dl)
    finally:
        backend.scene_destroy(hd)
    assert clamp > 0 and np.any(want != whole)
    tol = 20 * w * h * 2.0 ** -24 * np.abs(whole).max(axis=0, keepdims=True)
    assert np.all(np.abs(got - want) <= tol)


def test_more_materials_than_the_blocks_sums_hold(backend, oracle):
    """1,024 materials fill the 32 KB of a block's sums; with 1,025 they go to
    the gradient directly.  Both give the same gradient: at most 2,000 additions
    of either order, 2^-24 each, on sums without much cancellation."""
    torch = _torch()
    d = _case(oracle)
    cfg = d["config"]
    dl = torch.linspace(0.1, 1.0, cfg.width * cfg.height * 3, device="cuda")
    grads = []
    for n in (1024, 1025):
        p = np.zeros((n, 8), np.float32)
        p[: len(d["params"])] = d["params"]
        e = dict(d, params=p)
        h = backend.scene_create(d["scene"])
        try:
            _set(backend, h, e, p)
            grads.append(_grad(backend, h, e, 5, dl))
        finally:
            backend.scene_destroy(h)
    a, b = grads[0], grads[1][:1024]
    assert np.any(a != 0)
    assert np.all(np.abs(a - b) <= 2000 * 2.0 ** -24 * np.abs(a).max(axis=0, keepdims=True) + 1e-12)
    assert not np.any(grads[1][1024])
