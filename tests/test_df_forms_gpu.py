"""svo-df's two masked forms, the warp walk and one ray per lane, and the rule
between them: the same pixels, emission and word counts on trees of every small
depth, at regions that leave warps partly idle, and on both sides of the rule's
line (a pixel at the octree's centre as wide as the smallest leaf), as a frame,
in a batch and in a batch graph."""
from __future__ import annotations

import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("side", [2, 3, 4, 7, 16, 33])
@pytest.mark.parametrize("size", [(1, 1), (9, 5), (37, 41)])
def test_df_forms_are_identical(ctx, monkeypatch, side, size):
    import torch
    import xenodon_gb300 as xg
    from xenodon_gb300 import cameras, volumes
    g = volumes.random_grid(side, side, side, seed=side, density=0.5, levels=5)
    nodes, st = ctx.build_svo(g, "sparse")
    vol = ctx.upload_svo(nodes, st["side"])
    w, h = size
    p = xg.make_params(w, h, 3.0)
    # far away, near, and inside the octree
    for cam_t in (cameras.look_at((0.9, 1.3, -9.0), (0.5, 0.5, 0.5)), cameras.look_at((-0.4, 0.3, 1.9), (0.5, 0.4, 0.5)),
                  cameras.look_at((0.4, 0.45, 0.5), (0.9, 0.1, 0.7))):
        cam = xg.make_camera(*cam_t)
        got = []
        for form in (None, "1", "0"):
            if form is None:
                monkeypatch.delenv("XN_DF_PACKET", raising=False)
            else:
                monkeypatch.setenv("XN_DF_PACKET", form)
            rgba = torch.zeros((h, w, 4), dtype=torch.uint8, device="cuda")
            em = torch.zeros((h, w, 3), dtype=torch.float32, device="cuda")
            loads = torch.zeros((h, w), dtype=torch.int32, device="cuda")
            ctx.render_device(vol, "svo-df", cam, p, rgba.data_ptr(), em.data_ptr(), loads.data_ptr())
            plain = torch.zeros_like(rgba)
            ctx.render_device(vol, "svo-df", cam, p, plain.data_ptr())
            batch = torch.zeros((2, h, w, 4), dtype=torch.uint8, device="cuda")
            jobs = ctx.make_jobs([(vol, "svo-df", cam, p, batch[0].data_ptr())])
            ctx.render_batch(jobs, 1)
            graph = ctx.batch_graph(2)
            jobs = ctx.make_jobs([(vol, "svo-df", cam, p, batch[1].data_ptr())])
            graph.launch(jobs, 1)
            torch.cuda.synchronize()
            graph.close()
            got.append([t.cpu().numpy() for t in (rgba, em, loads, plain, batch[0], batch[1])])
        for k in (1, 2):
            for x, y in zip(got[0], got[k]):
                assert np.array_equal(x, y)
        for k in (3, 4, 5):
            assert np.array_equal(got[0][0], got[0][k])
        ref = oracle.render("svo-df", nodes=nodes, camera=oracle.make_camera(*cam_t), view=oracle.make_view(w, h, 3.0))
        assert np.array_equal(got[0][0], ref["rgba"])
    vol.release()


def test_df_rule_follows_the_pixel_width(ctx):
    """The same camera at two resolutions, one on each side of the line: the
    fine frame's pixels at the coarse frame's sample points are the same."""
    import xenodon_gb300 as xg
    from xenodon_gb300 import cameras, volumes
    g = volumes.random_grid(32, 32, 32, seed=4, density=0.4, levels=4)
    nodes, st = ctx.build_svo(g, "sparse")
    vol = ctx.upload_svo(nodes, st["side"])
    cam = xg.make_camera(*cameras.look_at((0.7, 0.9, -1.2), (0.5, 0.5, 0.5)))
    n = 8
    while n <= 256:  # 32 leaves across: pixel widths of 7 down to 0.2 leaves
        fine, _, _ = ctx.render(vol, "svo-df", cam, xg.make_params(2 * n, 2 * n, 2.0))
        coarse, _, _ = ctx.render(vol, "svo-df", cam, xg.make_params(n, n, 2.0))
        assert np.array_equal(fine[::2, ::2], coarse)
        n *= 2
    vol.release()
