"""The octree build over 16^3-voxel bricks at the sizes where it can go wrong:
the smallest sides it takes, sides just below and above a brick and a power of
two, thin grids, rows that 16-byte loads cannot read, uniform and partly
uniform bricks, and trees whose levels above the bricks need several launches.
Whole numbers throughout: every comparison is exact."""
from __future__ import annotations

import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu

# (dz, dy, dx)
SHAPES = [(16, 16, 16), (9, 1, 1), (1, 17, 2), (16, 16, 20), (15, 17, 33), (33, 31, 16), (1, 1, 70), (3, 64, 5),
          (40, 50, 24), (65, 18, 31)]


def _grid(shape, seed):
    """Random voxels at a density that leaves uniform cells of every size, with
    uniform blocks of 4, 8 and 16 voxels and a varied alpha."""
    from xenodon_gb300 import volumes
    rng = np.random.default_rng(seed)
    g = volumes.random_grid(*shape, seed=seed, density=float(rng.uniform(0.02, 0.6)), levels=4)
    if seed % 2:
        g[..., 3] = rng.integers(200, 256, shape)
    for e in (4, 8, 16):
        for _ in range(6):
            z, y, x = (int(rng.integers(0, max(1, d // e))) * e for d in shape)
            g[z:z + e, y:y + e, x:x + e] = rng.integers(0, 256, 4)
    return g


@pytest.mark.parametrize("heuristic,threshold", [("chan-diff", 0), ("chan-diff", 90), ("std-dev", 0.0),
                                                 ("std-dev", 40.0)])
@pytest.mark.parametrize("svo_type", ["sparse", "rope"])
@pytest.mark.parametrize("shape", SHAPES)
def test_brick_build_matches_oracle(ctx, shape, svo_type, heuristic, threshold):
    for seed in (1, 2):
        g = _grid(shape, seed)
        ref, rstats = oracle.build_svo(g, svo_type, heuristic, threshold)
        got, stats = ctx.build_svo(g, svo_type, heuristic, threshold)
        assert stats == rstats
        assert np.array_equal(got, ref)


@pytest.mark.parametrize("svo_type", ["sparse", "rope"])
@pytest.mark.parametrize("shape", SHAPES + [(300, 7, 290)])
def test_brick_layout_matches_upload(ctx, tmp_path, shape, svo_type):
    """The device layout written by the build, byte for byte the one made from
    the node array; the lean form its internal nodes; and the grid on the
    device at an address that 16-byte loads cannot use."""
    import torch
    g = _grid(shape, 3)
    dims = (shape[2], shape[1], shape[0])
    nodes, stats = ctx.build_svo(g, svo_type)
    up = ctx.upload_svo(nodes, stats["side"])
    buf = torch.zeros(g.size // 4 + 1, dtype=torch.int32, device="cuda")
    buf[1:] = torch.from_numpy(g.reshape(-1).view(np.int32)).cuda()
    torch.cuda.synchronize()
    built, bstats = ctx.build_svo_volume(buf.data_ptr() + 4, dims, svo_type)
    assert bstats == stats
    up.save(tmp_path / "up.svc")
    built.save(tmp_path / "built.svc")
    a, b = ((tmp_path / n).read_bytes() for n in ("up.svc", "built.svc"))
    if svo_type == "sparse":
        lean, lstats = ctx.build_svo_volume(buf.data_ptr() + 4, dims, "sparse", lean=True)
        assert lstats == stats
        lean.save(tmp_path / "lean.svc")
        again = ctx.load_volume(tmp_path / "lean.svc")
        assert again.info()["n_nodes"] == stats["n_nodes"]
    if stats["n_nodes"] == 1:  # a leaf root has no ropes to find: the flag of a build is its type's
        a, b = a[:12] + a[16:], b[:12] + b[16:]
    assert a == b


@pytest.mark.parametrize("side", [48, 272])
def test_brick_levels_above(ctx, side):
    """Uniform regions larger than a brick (leaves above the bricks, with ropes
    across levels), and with 272 a level above the bricks of more cells than
    one block takes."""
    rng = np.random.default_rng(side)
    shape = (side, side - 16, side)
    g = np.zeros(shape + (4,), np.uint8)
    g[..., 3] = 255
    for _ in range(40):
        z, y, x = (int(rng.integers(0, d)) for d in shape)
        g[z:z + 9, y:y + 5, x:x + 7] = rng.integers(0, 256, 4)
    for heuristic, threshold in (("chan-diff", 0), ("std-dev", 3.0)):
        ref, rstats = oracle.build_svo(g, "rope", heuristic, threshold)
        got, stats = ctx.build_svo(g, "rope", heuristic, threshold)
        assert stats == rstats
        assert np.array_equal(got, ref)
