"""Frames captured into a CUDA graph: a context that has rendered a frame of the
same size needs no memory and no wait for a plain frame of any other sample count,
so the frame can be captured; its replay gives the frame."""
import pytest

from raymotion_b200 import Backend, RenderConfig, _abi
from raymotion_b200.scenes import sized_field

pytestmark = pytest.mark.gpu


def _cfg(spp, adapt):
    c = RenderConfig(width=320, height=180, spp=spp, max_bounces=4, restir_candidates=1, restir_spatial=0,
                     flags=_abi.RM_FLAG_NO_ENV | _abi.RM_FLAG_DENOISE_OFF)
    c.adapt_min, c.adapt_step = adapt
    return c


# one lane; 8 lanes and segments; more than eight segments; 32 lanes
CASES = [(4, (16, 8)), (24, (16, 8)), (256, (16, 8)), (64, (0, 8))]


@pytest.mark.parametrize("warm", [None, 1, 24], ids=["same", "after_1spp", "after_24spp"])
@pytest.mark.parametrize("spp,adapt", CASES)
def test_plain_frames(backend, spp, adapt, warm):
    import torch
    sb, cam, _ = sized_field(5, 3000, 64, 36, 1, 4)
    sc = sb.pack()
    out = torch.empty(320 * 180 * 3, device="cuda")
    b = Backend(0)
    scene = b.scene_create(sc)
    try:
        # (every kernel is loaded by a context of its own)
        other = backend.scene_create(sc)
        for s, a in [*CASES, (24, (16, 8))]:
            backend.render_scene_async(other, cam, _cfg(s, a), 5, None, out.data_ptr())
        small = _cfg(64, (32, 32))
        small.width, small.height = 32, 18
        backend.render_scene_async(other, cam, small, 5, None, out.data_ptr())
        small.spp, small.adapt_min, small.adapt_step = 24, 16, 8
        backend.render_scene_async(other, cam, small, 5, None, out.data_ptr())
        backend.render_scene_async(other, cam, _cfg(spp, adapt), 5, None, out.data_ptr())
        backend.sync()
        backend.scene_destroy(other)
        want = out.clone()
        stream = torch.cuda.Stream()
        b.set_stream(stream.cuda_stream)
        # the frame's own images, which every call needs: by a frame of the same size
        b.render_scene_async(scene, cam, _cfg(warm or 1, (16, 8)), 5, None, out.data_ptr())
        if warm is None:
            b.render_scene_async(scene, cam, _cfg(spp, adapt), 5, None, out.data_ptr())
        b.sync()
        out.zero_()
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream, capture_error_mode="thread_local"):
            b.render_scene_async(scene, cam, _cfg(spp, adapt), 5, None, out.data_ptr())
        for _ in range(2):
            out.zero_()
            torch.cuda.synchronize()
            graph.replay()
            torch.cuda.synchronize()
            assert torch.equal(out.view(torch.int32), want.view(torch.int32))
        del graph
    finally:
        torch.cuda.synchronize()
        b.scene_destroy(scene)
        b.close()


@pytest.mark.parametrize("spp,adapt", CASES)
def test_graphs_outlive_larger_frames(backend, spp, adapt):
    """A graph keeps the workspace that it was captured with: a frame that needs a
    larger one, and another context that takes freed memory, change nothing."""
    import torch
    sb, cam, _ = sized_field(5, 3000, 64, 36, 1, 4)
    sc = sb.pack()
    out, other_out = (torch.empty(320 * 180 * 3, device="cuda") for _ in range(2))
    b, other = Backend(0), None
    scene = b.scene_create(sc)
    try:
        stream = torch.cuda.Stream()
        b.set_stream(stream.cuda_stream)
        b.render_scene_async(scene, cam, _cfg(spp, adapt), 5, None, out.data_ptr())
        b.sync()
        want = out.clone()
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream, capture_error_mode="thread_local"):
            b.render_scene_async(scene, cam, _cfg(spp, adapt), 5, None, out.data_ptr())
        b.render_scene_async(scene, cam, _cfg(320, (0, 8)), 6, None, out.data_ptr())
        b.sync()
        other = Backend(0)
        theirs = other.scene_create(sc)
        other.render_scene_async(theirs, cam, _cfg(64, (0, 8)), 7, None, other_out.data_ptr())
        other.sync()
        other_want = other_out.clone()
        out.zero_()
        torch.cuda.synchronize()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(out.view(torch.int32), want.view(torch.int32))
        other.render_scene_async(theirs, cam, _cfg(64, (0, 8)), 7, None, other_out.data_ptr())
        other.sync()
        assert torch.equal(other_out.view(torch.int32), other_want.view(torch.int32))
        other.scene_destroy(theirs)
        del graph
    finally:
        torch.cuda.synchronize()
        b.scene_destroy(scene)
        b.close()
        if other:
            other.close()


def test_gradients_of_two_graphs_at_the_same_time(backend):
    """Two captured gradients hand out their pixel lanes apart from one another.
    Rounding: the order of the additions, 2^-20 of the largest entry."""
    import numpy as np
    import torch

    from raymotion_b200.scenes import inverse_scene
    d = inverse_scene(4, n_spheres=10, n_dielectric=3, ground=20, width=128, height=128, spp=8, depth=5)
    scene = backend.scene_create(d["scene"])
    try:
        backend.scene_set_materials(scene, d["params"], d["tri_material"])
        dl = [torch.rand(128 * 128 * 3, device="cuda", generator=torch.Generator("cuda").manual_seed(k)) for k in (1, 2)]
        grad = [torch.zeros(len(d["params"]) * 8, device="cuda") for _ in range(2)]
        streams = [torch.cuda.Stream() for _ in range(2)]
        want, graphs = [], []
        for k in range(2):
            backend.set_stream(streams[k].cuda_stream)
            torch.cuda.synchronize()
            backend.backward(scene, d["camera"], d["config"], 5 + k, dl[k].data_ptr(), grad[k].data_ptr())
            backend.sync()
            want.append(grad[k].cpu().numpy())
            g = torch.cuda.CUDAGraph()
            with torch.cuda.graph(g, stream=streams[k], capture_error_mode="thread_local"):
                backend.backward(scene, d["camera"], d["config"], 5 + k, dl[k].data_ptr(), grad[k].data_ptr())
            graphs.append(g)
        for _ in range(4):
            for k in range(2):
                grad[k].zero_()
            torch.cuda.synchronize()
            for k in range(2):
                with torch.cuda.stream(streams[k]):
                    graphs[k].replay()
            torch.cuda.synchronize()
            for k in range(2):
                assert np.abs(grad[k].cpu().numpy() - want[k]).max() <= 2.0 ** -20 * np.abs(want[k]).max()
        del graphs
    finally:
        torch.cuda.synchronize()
        backend.set_stream(None)
        backend.scene_destroy(scene)


def _scenes_beside(backend_of_thread, sc, rounds):
    """Create, grow and give back scenes in another thread; its errors."""
    import threading
    errors = []

    def work():
        try:
            for _ in range(rounds):
                h = backend_of_thread.scene_create(sc)
                backend_of_thread.scene_destroy(h)
        except Exception as e:  # noqa: BLE001
            errors.append(e)
    t = threading.Thread(target=work)
    t.start()
    return t, errors


def test_memory_given_back_beside_a_capture(backend):
    """Another thread's scenes come and go while this one captures a frame."""
    import torch
    sb, cam, _ = sized_field(5, 3000, 64, 36, 1, 4)
    sc = sb.pack()
    out = torch.empty(320 * 180 * 3, device="cuda")
    b = Backend(0)
    scene = backend.scene_create(sc)
    try:
        stream = torch.cuda.Stream()
        backend.set_stream(stream.cuda_stream)
        backend.render_scene_async(scene, cam, _cfg(4, (16, 8)), 5, None, out.data_ptr())
        backend.sync()
        want = out.clone()
        out.zero_()
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream, capture_error_mode="thread_local"):
            backend.render_scene_async(scene, cam, _cfg(4, (16, 8)), 5, None, out.data_ptr())
            t, errors = _scenes_beside(b, sc, 3)
            t.join()
        assert not errors
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(out, want)
        del graph
    finally:
        torch.cuda.synchronize()
        backend.set_stream(None)
        backend.scene_destroy(scene)
        b.close()


def test_memory_given_back_beside_batches(backend):
    """The batch's pool captures its waves; another context's scenes come and go."""
    import torch

    from raymotion_b200 import BatchItem
    sb, cam, _ = sized_field(5, 3000, 64, 36, 1, 4)
    sc = sb.pack()
    cfg = _cfg(4, (0, 8))
    cfg.width, cfg.height = 32, 18
    b = Backend(0)
    scene = backend.scene_create(sc)
    outs = [torch.empty(32 * 18 * 3, device="cuda") for _ in range(40)]
    items = [BatchItem(scene, cam, cfg, 9, None, o.data_ptr(), None) for o in outs]
    try:
        t, errors = _scenes_beside(b, sc, 60)
        while t.is_alive():
            for o in outs:
                o.zero_()
            torch.cuda.synchronize()
            backend.render_batch(items)
            assert len(backend.batch_log()) > 0
            assert all(torch.equal(o, outs[0]) for o in outs) and outs[0].any()
        t.join()
        assert not errors
    finally:
        backend.scene_destroy(scene)
        b.close()
