"""Macrocell codes of scenes whose bricks differ much in size (the codes' CTAs are
shared out by size): frames and sample counts equal the oracle's for several
transfer functions."""
import numpy as np
import pytest

from aloha_gb300 import scenes as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims,cuts", [
    ((300, 24, 20), ([4, 8, 12, 20, 21, 290], [], [])),  # slivers beside one long brick
    ((66, 70, 62), ([1, 33], [5, 61], [2])),
    ((1030, 5, 6), ([], [], [])),  # rows beyond one CTA's cells
    ((9, 8, 520), ([], [], [8])),
])
def test_uneven_bricks(gpu_ctx_factory, oracle, dims, cuts):
    rng = np.random.default_rng(sum(dims))
    nx, ny, nz = dims
    vol = (0.15 * rng.random((nz, ny, nx))).astype(np.float32)
    spikes = max(3, nx * ny * nz // 3000)
    at = tuple(rng.integers(0, n, spikes) for n in (nz, ny, nx))
    vol[at] = rng.uniform(0.3, 1.0, spikes).astype(np.float32)
    descs = S.grid_split(dims, cuts)
    vox = S.extract_bricks(vol, descs)
    W, H = 96, 64
    ctx = gpu_ctx_factory()
    ctx.set_bricks(descs, vox)
    ctx.set_ranks(1)
    ctx.set_params()
    cam = S.orbit_cameras(dims, 1, W, H, seed=113, distance=0.9)[0]
    ctx.set_camera(0, *cam)
    ctx.resize(0, W, H)
    low = S.ramp_tf()
    low[:30, 3] = 0.02
    high = S.ramp_tf()
    high[:200, 3] = 0.0
    for tf in (S.ramp_tf(), low, high, S.ramp_tf(16)):
        ctx.set_transfer_function(tf)
        ref = oracle.render(descs, vox, tf, oracle.make_camera(*cam), W, H, oracle.make_params(), n_ranks=1)
        np.testing.assert_array_equal(ctx.render(0, width=W, height=H), ref["fb"])
        assert ctx.stats().samples == ref["samples"]
