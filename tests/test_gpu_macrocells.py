"""Brick upload and macrocell codes at their edges: volumes whose rows end
around the upload kernel's column chunks, thinner than a macrocell, and empty
but for scattered voxels, so that rays step over boxes of many cells next to
full ones.  Frames and sample counts must equal the oracle's, which evaluates
every sample."""
import numpy as np
import pytest

from aloha_gb300 import abi
from aloha_gb300 import scenes as S
from aloha_gb300 import volfile as V

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims,bricks", [
    ((119, 9, 12), 1), ((120, 13, 10), 1), ((121, 17, 8), 1), ((125, 8, 16), 1), ((244, 5, 7), 1), ((251, 6, 9), 1),
    ((3, 2, 5), 1), ((4, 4, 4), 1), ((5, 1, 70), 1), ((1, 40, 33), 1), ((70, 66, 68), 1), ((70, 66, 68), 7),
    ((40, 90, 33), 33)])
@pytest.mark.parametrize("kw", [{}, dict(dt=0.3, jitter_mode=abi.JITTER_NONE)])
def test_sparse_volumes(gpu_ctx_factory, oracle, dims, bricks, kw):
    rng = np.random.default_rng(sum(dims) + bricks)
    nx, ny, nz = dims
    vol = (0.15 * rng.random((nz, ny, nx))).astype(np.float32)  # below the ramp's first visible value
    spikes = max(2, nx * ny * nz // 4000)
    vol[rng.integers(0, nz, spikes), rng.integers(0, ny, spikes), rng.integers(0, nx, spikes)] = 0.9
    descs = S.single_brick(dims) if bricks == 1 else V.chopsuey_split(dims, bricks)
    vox = S.extract_bricks(vol, descs)
    tf = S.ramp_tf()
    W, H = 90, 70
    ctx = gpu_ctx_factory()
    ctx.set_bricks(descs, vox)
    ctx.set_transfer_function(tf)
    ctx.set_params(**kw)
    for v, cam in enumerate(S.orbit_cameras(dims, 2, W, H, seed=79, distance=1.1)):
        ctx.set_camera(v, *cam)
        ctx.resize(v, W, H)
        ref = oracle.render(descs, vox, tf, oracle.make_camera(*cam), W, H, oracle.make_params(**kw),
                            n_ranks=len(descs))
        np.testing.assert_array_equal(ctx.render(v, width=W, height=H), ref["fb"])
        assert ctx.stats().samples == ref["samples"]
    # other entries become visible: the codes follow the transfer function
    tf2 = tf.copy()
    tf2[:20, 3] = 0.05
    ctx.set_transfer_function(tf2)
    ref = oracle.render(descs, vox, tf2, oracle.make_camera(*cam), W, H, oracle.make_params(**kw), n_ranks=len(descs))
    np.testing.assert_array_equal(ctx.render(1, width=W, height=H), ref["fb"])
