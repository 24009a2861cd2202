"""Small frames, traced by warps of fewer rays: regions of one display rendered
alone (sizes at the edges of 2x1, 2x2, 4x2 and 4x4 pixel warps and of the rules
that choose them) against the same pixels of the whole frame, which is traced
by full warps; image, emission and word counts."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

W, H = 700, 600
# the most rays that warps of 2, 4, 8 and 16 take on 152 SMs: from inside 2432,
# 4864, 9728 and 19456; outside 7296, 14592, 29184 and 58368 in small volumes,
# twice that in large ones
SIZES = [(1, 1), (3, 5), (17, 9), (49, 49), (50, 49), (76, 64), (77, 64), (85, 85), (86, 85), (120, 121), (121, 121),
         (139, 139), (140, 140), (170, 171), (171, 171), (241, 242), (242, 242), (341, 342), (342, 342)]


@pytest.mark.parametrize("trav", ["dda", "svo-naive", "esvo", "svo-df", "svo-rope"])
@pytest.mark.parametrize("where", ["outside", "inside"])
@pytest.mark.parametrize("dims", [(40, 33, 40), (132, 20, 17)])  # a small volume and one that counts as large
def test_regions_match_the_whole_frame(ctx, trav, where, dims):
    import torch
    import xenodon_gb300 as xg
    from xenodon_gb300 import cameras, volumes
    g = volumes.random_grid(*dims[::-1], seed=8, density=0.35, levels=6)
    if trav == "dda":
        vol, c = ctx.upload_grid(g), cameras.volume_centre(dims)
    else:
        nodes, st = ctx.build_svo(g, "rope")
        vol, c = ctx.upload_svo(nodes, st["side"]), np.array(dims) / (2 * st["side"])
    pos = c + np.array([0.5, 0.4, -1.5]) * (1.0 if where == "outside" else 0.1)
    cam = xg.make_camera(*cameras.look_at(pos, c))

    def render(w, h, offset):
        p = xg.make_params(w, h, 2.0, output_offset=offset, display_extent=(W, H))
        rgba = torch.zeros((h, w, 4), dtype=torch.uint8, device="cuda")
        em = torch.zeros((h, w, 3), dtype=torch.float32, device="cuda")
        loads = torch.zeros((h, w), dtype=torch.int32, device="cuda")
        ctx.render_device(vol, trav, cam, p, rgba.data_ptr(), em.data_ptr(), loads.data_ptr())
        plain = torch.zeros_like(rgba)
        ctx.render_device(vol, trav, cam, p, plain.data_ptr())
        torch.cuda.synchronize()
        return [t.cpu().numpy() for t in (rgba, em, loads, plain)]

    whole = render(W, H, (0, 0))
    assert whole[0][..., :3].any()
    for w, h in SIZES:
        x, y = (W - w) // 2 + 1, (H - h) // 3
        for part, full in zip(render(w, h, (x, y)), whole):
            assert np.array_equal(part, full[y:y + h, x:x + w]), (w, h)
    vol.release()
