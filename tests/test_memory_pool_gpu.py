"""Freed device memory kept by a context: builds and uploads of about the same
size give the same trees on reused memory, a budget is never exceeded by it,
volumes released while another stream renders them stay intact, and several
threads may build and release at once."""
from __future__ import annotations

import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _grid(seed):
    from xenodon_gb300 import volumes
    return volumes.random_grid(60, 50, 72, seed=seed, density=0.4, levels=7)


def test_reused_memory_gives_the_same_trees(ctx):
    import torch
    import xenodon_gb300 as xg
    from xenodon_gb300 import cameras
    cam = xg.make_camera(*cameras.look_at((1.3, 0.9, -1.0), (0.28, 0.2, 0.23)))
    p = xg.make_params(200, 150, 2.0)
    used0 = ctx.memory()[0]
    frames = {}
    for turn in range(3):
        for seed in (1, 2, 3):
            d = torch.from_numpy(_grid(seed)).cuda()
            torch.cuda.synchronize()
            vol, _ = ctx.build_svo_volume(d.data_ptr(), (72, 50, 60), "rope")
            out = torch.zeros((4, 150, 200, 4), dtype=torch.uint8, device="cuda")
            stream = torch.cuda.Stream()
            stream.wait_stream(torch.cuda.current_stream())
            for k, t in enumerate(xg.SVO_TRAVERSALS):
                ctx.render_device(vol, t, cam, p, out[k].data_ptr(), None, None, stream.cuda_stream)
            vol.release()  # the renders may still run
            ctx.build_svo_volume(d.data_ptr(), (72, 50, 60), "sparse", lean=True)[0].release()
            torch.cuda.synchronize()
            got = out.cpu().numpy()
            assert got[..., :3].any()
            assert np.array_equal(frames.setdefault(seed, got), got)
    assert ctx.memory()[0] == used0


def test_pool_stays_within_the_budget(built_library):
    import torch
    import xenodon_gb300 as xg
    g = _grid(4)
    with xg.Context(0, hbm_budget=96 << 20) as c:
        for _ in range(3):
            nodes, stats = c.build_svo(g, "rope")
            vol = c.upload_svo(nodes, stats["side"])
            assert c.memory()[0] <= 96 << 20
            vol.release()
        # the whole budget can still be taken by one volume
        big = np.zeros((80, 512, 512, 4), np.uint8)
        vol = c.upload_grid(big)
        assert vol.info()["device_bytes"] == big.nbytes
        vol.release()
        with pytest.raises(xg.XenodonError) as e:
            c.upload_grid(np.zeros((100, 512, 512, 4), np.uint8))
        assert e.value.code == xg.XN_ERR_BUDGET
    torch.cuda.synchronize()


def test_threads_build_and_release(ctx):
    ref = {s: ctx.build_svo(_grid(s), "rope")[0] for s in (5, 6, 7)}
    bad = []

    def work(seed):
        g = _grid(seed)
        for _ in range(5):
            if not np.array_equal(ctx.build_svo(g, "rope")[0], ref[seed]):
                bad.append(seed)

    threads = [threading.Thread(target=work, args=(s,)) for s in ref]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad
