"""Calls on a device whose memory is almost taken.

What a call keeps only for speed it does without there, and its outputs stay the
same: the plain frame and the batch take smaller chunks of samples or the lane
kernels (rm_paths.cu, rm_kernels.cu), a small ReSTIR frame draws its candidates a
thread a pixel instead of in tiles (rm_kernels.cu), and a new upload of a scene
checks the triangles before they take the place of the old ones, instead of beside
them.

A child process makes its scenes, runs every call once at a small size, takes
the device's memory but for 4, 48 and 160 MB with one tensor and runs the calls each
time, gives the tensor back and runs them again."""
import os
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu

CHILD = '''
import sys
import numpy as np, torch
import raymotion_b200 as rb
from raymotion_b200 import BatchItem, RenderConfig, _abi
from raymotion_b200.scenes import PLAIN_FLAGS, sized_field

WHAT = sys.argv[1]
W, H = 1280, 720
b = rb.Backend(0)
sb, cam, _ = sized_field(5, 3000, 64, 36, 1, 4)
scene = b.scene_create(sb.pack())


def cfg(spp, w=W, h=H, adapt=0):
    c = RenderConfig(width=w, height=h, spp=spp, max_bounces=3, restir_candidates=1, restir_spatial=0, flags=PLAIN_FLAGS)
    c.adapt_min, c.adapt_step = adapt, 8 if spp < 32 else 32
    return c


hdr = [torch.empty(W * H * 3, device="cuda") for _ in range(3)]


def frame(c, k=0):
    hdr[k].zero_()
    torch.cuda.synchronize()
    b.render_scene_async(scene, cam, c, 7, None, hdr[k].data_ptr())
    b.sync()
    return hdr[k].cpu().numpy().copy()


def batch(c):
    b.render_batch([BatchItem(scene, cam, c, 30 + k, None, hdr[k].data_ptr(), None) for k in range(3)])
    b.sync()
    return np.stack([x.cpu().numpy() for x in hdr])


def restir(w, h):
    c = RenderConfig(width=w, height=h, spp=1, max_bounces=3, restir_candidates=8, restir_spatial=2, adapt_min=0,
                     flags=_abi.RM_FLAG_NO_ENV)
    b.reset_history()
    return frame(c)


def soup(n, seed):
    from raymotion_b200.scene import SceneBuilder
    r = np.random.default_rng(seed)
    c = r.uniform(-20, 20, (n, 3)).astype(np.float32)
    s = SceneBuilder()
    s.add_triangles(c, c + r.normal(0, 0.3, (n, 3)), c + r.normal(0, 0.3, (n, 3)))
    return s.pack()


if WHAT == "upload":  # 70 MB of triangles; fewer; as many; one with a texture that is not there
    scenes = [soup(400000, 1), soup(399000, 2), soup(399000, 3), soup(399000, 4)]
    scenes[3].tris["texture_offset"][398999] = 0
    r = np.random.default_rng(5)
    rays = np.concatenate([r.uniform(-20, 20, (4096, 3)), r.normal(size=(4096, 3)), np.full((4096, 1), 50)], 1)
    rays = torch.from_numpy(rays.astype(np.float32)).cuda()
    tri = torch.empty(4096, dtype=torch.int32, device="cuda")

    def hits():
        b.trace(rays.data_ptr(), 4096, False, tri.data_ptr())
        return tri.cpu().numpy() + 1  # (0: a miss)

    def uploads():
        out = []
        for s in scenes[:3]:
            b.upload(s, use_nodes=False)
            out.append(hits())
        try:
            b.upload(scenes[3], use_nodes=False)
            raise SystemExit("accepted")
        except rb.RenderError as e:
            assert "texture" in str(e), e
        return out + [hits()]

    b.upload(scenes[0], use_nodes=False)
    hits()
if WHAT == "restir":
    restir(W, H)
frame(cfg(1))  # the frame's own buffers at their size
for c in (cfg(8, 32, 18, 8), cfg(24, 32, 18, 8), cfg(64, 32, 18, 32), cfg(64, 32, 18), cfg(24, 320, 180, 8), cfg(64, 320, 180, 32)):
    frame(c)  # every kernel once
batch(cfg(16, 32, 18))
calls = {"frame": lambda: [frame(cfg(4)), frame(cfg(16)), frame(cfg(16, adapt=8)), frame(cfg(64))],
         "batch": lambda: [batch(cfg(16)), batch(cfg(3))], "restir": lambda: [restir(333, 187)],
         "upload": lambda: uploads()}[WHAT]
low = {}
for leave in (4, 48, 160):  # MB
    taken = torch.empty(torch.cuda.mem_get_info()[0] - (leave << 20), dtype=torch.uint8, device="cuda")
    low[leave] = calls()
    del taken
    torch.cuda.empty_cache()
full = calls()
assert all(x.any() for x in full)
for leave, out in low.items():
    assert all(np.array_equal(a.view(np.uint32), c.view(np.uint32)) for a, c in zip(out, full)), leave
print("the same")
'''


@pytest.mark.parametrize("what", ["frame", "batch", "restir", "upload"])
def test_outputs_do_not_depend_on_free_memory(what):
    root = Path(__file__).resolve().parents[1]
    r = subprocess.run([sys.executable, "-c", CHILD, what], capture_output=True, text=True, cwd=root,
                       env=dict(os.environ, PYTHONPATH=str(root)), timeout=300)
    assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-3000:]
    assert "the same" in r.stdout, r.stdout
