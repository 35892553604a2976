"""The all-empty segments' backward: two lanes per segment and copies of its
shared bins, whose number depends on the transfer function's size.  Sizes on
both sides of each line, with segments of odd, even and single samples (the
second lane's last sample is missing or not) against the oracle's adjoint."""
import numpy as np
import pytest

from aloha_gb300 import scenes as S
from aloha_gb300 import volfile as V
from tests import scenes_for_tests as T

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_tf,k,dt", [(2, 32, 0.5), (290, 32, 0.5), (291, 7, 0.5), (732, 7, 0.3), (733, 32, 0.3),
                                       (2044, 1, 0.5), (2045, 33, 0.5), (256, 1, 0.3), (256, 3, 0.5)])
@pytest.mark.parametrize("views", [1, 2])
def test_alpha_gradient(gpu_ctx_factory, oracle, n_tf, k, dt, views):
    dims, W, H = (37, 30, 41), 47, 38
    vol = S.blob_field(dims, 6, (2.0, 5.0), seed=57)
    descs = V.chopsuey_split(dims, 4)
    vox = S.extract_bricks(vol, descs)
    tf = S.ramp_tf(n_tf)
    ctx = gpu_ctx_factory()
    ctx.set_bricks(descs, vox)
    ctx.set_transfer_function(tf)
    ctx.set_ranks(1)
    ctx.set_params(dt=dt)
    cams = T.cameras(dims, views, W, H, seed=63)
    rng = np.random.default_rng(67)
    dls = [rng.uniform(-1, 1, (H, W, 4)).astype(np.float32) for _ in cams]
    ref = np.zeros((n_tf, 4))
    for v, cam in enumerate(cams):
        ctx.set_camera(v, *cam)
        ctx.resize(v, W, H)
        ref += oracle.adjoint(descs, vox, tf, oracle.make_camera(*cam), W, H, dls[v], (0, 0, 0), dims,
                              oracle.make_params(dt=dt))["dtf"]
    ids = list(range(views))
    ctx.forward_views(ids, [np.zeros((H, W, 4), np.float32) for _ in ids], k)
    samples = ctx.stats().samples
    dtf = np.zeros((n_tf, 4), np.float32)
    ctx.backward_views(ids, dls, dtf, None, None, None)
    assert ctx.stats().samples == samples
    assert np.linalg.norm(dtf - ref) <= 5e-4 * np.linalg.norm(ref)
