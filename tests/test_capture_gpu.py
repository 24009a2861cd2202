"""Volumes released and octrees built while a stream is being captured, and the
memory of a volume that a captured graph or a launch still in flight reads."""
from __future__ import annotations

import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

W, H = 320, 240


def _setup(ctx, seed=11):
    import xenodon_gb300 as xg
    from xenodon_gb300 import cameras, volumes
    g = volumes.random_grid(64, 64, 64, seed=seed, density=0.4, levels=6)
    cam = xg.make_camera(*cameras.look_at((1.4, 1.1, -1.3), (0.5, 0.5, 0.5)))
    return g, cam, xg.make_params(W, H, 3.0)


@pytest.mark.parametrize("mode,thread", [("thread_local", "other"), ("relaxed", "other"), ("relaxed", "same")])
def test_release_and_build_leave_a_capture_valid(ctx, mode, thread):
    import torch
    import xenodon_gb300 as xg
    g, cam, p = _setup(ctx)
    nodes, st = ctx.build_svo(g, "rope")
    vol = ctx.upload_svo(nodes, st["side"])
    want, _, _ = ctx.render(vol, "esvo", cam, p)
    errors = []
    with xg.Context(0) as other:
        mine = other.upload_svo(nodes, st["side"])

        def work():
            try:
                mine.release()
                v, _ = other.build_svo_volume(g.ctypes.data, (64, 64, 64), "rope")
                v.release()
                assert np.array_equal(other.build_svo(g, "rope")[0], nodes)
            except Exception as e:  # reported by the capturing thread
                errors.append(e)

        s = torch.cuda.Stream()
        out = torch.zeros((H, W, 4), dtype=torch.uint8, device="cuda")
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=s, capture_error_mode=mode):
            ctx.render_device(vol, "esvo", cam, p, out.data_ptr(), None, None, s.cuda_stream)
            if thread == "same":
                work()
            else:
                t = threading.Thread(target=work)
                t.start()
                t.join()
        assert not errors
        graph.replay()
        torch.cuda.synchronize()
    assert np.array_equal(out.cpu().numpy(), want)
    vol.release()


@pytest.mark.parametrize("how", ["stream", "graph", "batch", "many streams"])
def test_a_released_volume_outlives_its_launches(ctx, how):
    """The volume is released, and its memory asked for again, while launches
    that read it are queued behind others."""
    import torch
    import xenodon_gb300 as xg
    g, cam, p = _setup(ctx)
    h, _, _ = _setup(ctx, seed=12)
    d = torch.from_numpy(h).cuda()
    keep, _ = ctx.build_svo_volume(d.data_ptr(), (64, 64, 64), "rope")
    nodes, st = ctx.build_svo(g, "rope")
    ref = ctx.upload_svo(nodes, st["side"])
    want, _, _ = ctx.render(ref, "svo-df", cam, p)
    ref.release()
    big = xg.make_params(1600, 1200, 3.0)
    for _ in range(3):
        vol = ctx.upload_svo(nodes, st["side"])
        # 64 streams that the context remembers, and some it does not
        streams = [torch.cuda.Stream() for _ in range(80 if how == "many streams" else 1)]
        s = streams[-1]
        raw = s.cuda_stream
        out = torch.zeros((H, W, 4), dtype=torch.uint8, device="cuda")
        dump = torch.zeros((1200, 1600, 4), dtype=torch.uint8, device="cuda")
        graph = torch.cuda.CUDAGraph()
        if how == "graph":
            with torch.cuda.graph(graph, stream=s):
                ctx.render_device(vol, "svo-df", cam, p, out.data_ptr(), None, None, raw)
        jobs = ctx.make_jobs([(vol, "svo-df", cam, p, out.data_ptr())])
        for x in streams[:-1]:
            ctx.render_device(keep, "svo-df", cam, p, dump.data_ptr(), None, None, x.cuda_stream)
        torch.cuda.synchronize()
        for _ in range(20):
            ctx.render_device(keep, "svo-df", cam, big, dump.data_ptr(), None, None, raw)
        if how == "graph":
            with torch.cuda.stream(s):
                graph.replay()
        elif how == "batch":
            ctx.render_batch(jobs, 1, stream=raw)
        else:
            ctx.render_device(vol, "svo-df", cam, p, out.data_ptr(), None, None, raw)
        vol.release()
        again, _ = ctx.build_svo_volume(d.data_ptr(), (64, 64, 64), "rope")
        torch.cuda.synchronize()
        assert np.array_equal(out.cpu().numpy(), want)
        again.release()
    keep.release()
