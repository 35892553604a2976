"""A brick that fits 2^31 quads only with plain pitches (internal.h): what it
shows in its last voxels is what a small brick of those voxels shows."""
import numpy as np
import pytest

from aloha_gb300 import abi
from aloha_gb300 import scenes as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(1024, 1440, 1440), (256, 2860, 2860)])
def test_last_voxels_of_a_brick_at_the_limit(gpu_ctx_factory, dims):
    torch = pytest.importorskip("torch")
    n, W, H = 64, 160, 120
    corner = S.blob_field((n, n, n), 6, (4.0, 10.0), seed=107)
    corner[:3] = corner[:, :3] = corner[:, :, :3] = 0.0  # as in the voxels next to it
    corner = torch.from_numpy(corner).cuda()
    vol = torch.zeros(dims[::-1], device="cuda")
    vol[-n:, -n:, -n:] = corner
    lo = [d - n for d in dims]
    small = {k: list(v) for k, v in S.single_brick((n, n, n))[0].items()}
    for key in ("cell_lo", "cell_hi", "voxel_lo", "voxel_hi", "space_lo", "space_hi"):
        small[key] = [v + o for v, o in zip(small[key], lo)]
    cam = S.orbit_cameras((n, n, n), 1, W, H, seed=109, distance=1.2)[0]
    cam = ((np.asarray(cam[0], np.float64) + lo).astype(np.float32),) + tuple(cam[1:])
    frames = []
    ctx = gpu_ctx_factory()
    for descs, vox in ((S.single_brick(dims), vol), ([small], corner)):
        ctx.set_bricks(descs, [vox])
        ctx.set_transfer_function(S.ramp_tf())
        ctx.set_params(jitter_mode=abi.JITTER_NONE)  # both bricks sample the same lattice of t
        ctx.set_camera(0, *cam)
        ctx.resize(0, W, H)
        frames.append(ctx.render(0, width=W, height=H).view(np.uint8).astype(int))
    ctx.close()
    # positions round at 2^-12 voxel in one brick and finer in the other: a value
    # differs by some 1e-4, a channel by at most 1.4e-2 over 200 samples that all
    # round the same way, and by a tenth of that otherwise
    assert (frames[1] > 0).mean() > 0.1
    assert np.abs(frames[0] - frames[1]).max() <= 4
    assert np.abs(frames[0] - frames[1]).mean() <= 0.2
