"""The generic batch form, one launch for a batch of any jobs, beside the forms
of single traversals: the same pixels, and no dearer than its dispatch."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(4, 256, 0, 0), (8, 128, 0, 2)])
def test_generic_form_beside_its_own(ctx, monkeypatch, shape):
    """esvo frames of a 256^3 gas field.  Measured in the time of esvo's own
    form: 1.05 to 1.15; with registers spilled for jobs that never reach the
    generic function 2.3 in the queue form."""
    import time
    import torch
    import xenodon_gb300 as xg
    from xenodon_gb300 import cameras, volumes
    n, frames = 256, 48
    d = torch.from_numpy(np.ascontiguousarray(volumes.gas_field(n, seed=2))).cuda()
    torch.cuda.synchronize()
    vol, _ = ctx.build_svo_volume(d.data_ptr(), (n, n, n), "sparse", lean=True)
    p = xg.make_params(256, 256, 2.0)
    out = torch.zeros((frames, 256, 256, 4), dtype=torch.uint8, device="cuda")
    c = np.array((0.5, 0.5, 0.5))
    jobs = ctx.make_jobs([
        (vol, "esvo", xg.make_camera(*cameras.look_at(c + 1.3 * np.array((np.cos(a), 0.23, np.sin(a))), c)), p, o.data_ptr())
        for a, o in zip(np.linspace(0, 6, frames), out)])

    def run():
        best = float("inf")
        for _ in range(6):
            torch.cuda.synchronize()
            t = time.perf_counter()
            ctx.render_batch(jobs, frames, xg.BatchConfig(*shape))
            torch.cuda.synchronize()
            best = min(best, time.perf_counter() - t)
        return best, out.cpu().numpy()

    own, image = run()
    out.zero_()
    monkeypatch.setenv("XN_BATCH_GENERIC", "1")
    generic, again = run()
    vol.release()
    assert image[..., :3].any() and np.array_equal(image, again)
    assert generic <= 1.6 * own, (generic, own)
