"""The transfer-function gradient of replayed samples, summed in as many shared
copies as the transfer function's size allows, on both sides of each line,
against the oracle's adjoint.  Smooth volumes: the lookup index mostly moves by
one entry and a pending sum moves along.  Noise: it jumps at every sample; a
sample's entry then depends on the rounding of its position, so with a constant
transfer function the sum over the entries is compared, which does not."""
import numpy as np
import pytest

from aloha_gb300 import scenes as S
from tests import scenes_for_tests as T

pytestmark = pytest.mark.gpu

SIZES = [2, 3, 64, 460, 461, 766, 767, 2048]


def gradients(make, oracle, vol, tf, density):
    dims, W, H = vol.shape[::-1], 44, 39
    descs = S.single_brick(dims)
    vox = S.extract_bricks(vol, descs)
    ctx = make()
    ctx.set_bricks(descs, vox)
    ctx.set_transfer_function(tf)
    ctx.set_ranks(1)
    ctx.set_params()
    cam = T.cameras(dims, 1, W, H, seed=79)[0]
    dl = np.random.default_rng(71).uniform(-1, 1, (H, W, 4)).astype(np.float32)
    ctx.set_camera(0, *cam)
    ctx.resize(0, W, H)
    ref = oracle.adjoint(descs, vox, tf, oracle.make_camera(*cam), W, H, dl, (0, 0, 0), dims, oracle.make_params())
    ctx.forward_views([0], [np.zeros((H, W, 4), np.float32)], 32)
    dtf = np.zeros(tf.shape, np.float32)
    dden = np.zeros(vol.shape, np.float32) if density else None
    ctx.backward_views([0], [dl], dtf, dden, *(((0, 0, 0), dims) if density else (None, None)))
    return dtf, ref["dtf"]


@pytest.mark.parametrize("n_tf", SIZES)
@pytest.mark.parametrize("density", [False, True])
def test_smooth(gpu_ctx_factory, oracle, n_tf, density):
    tf = S.ramp_tf(n_tf)
    tf[:, 3] = 0.01 + 0.1 * tf[:, 3]
    got, ref = gradients(gpu_ctx_factory, oracle, S.blob_field((29, 33, 26), 6, (2.0, 6.0), seed=73), tf, density)
    assert np.linalg.norm(got - ref) <= 5e-4 * np.linalg.norm(ref)


@pytest.mark.parametrize("n_tf", SIZES)
def test_noise_total(gpu_ctx_factory, oracle, n_tf):
    vol = np.random.default_rng(83).random((26, 33, 29)).astype(np.float32)
    tf = np.tile(np.array([[0.7, 0.4, 0.2, 0.05]], np.float32), (n_tf, 1))
    got, ref = gradients(gpu_ctx_factory, oracle, vol, tf, True)
    # a few hundred thousand fp32 terms of either sign: far below 1e-4 of their absolute sum
    assert np.all(np.abs(got.astype(np.float64).sum(0) - ref.sum(0)) <= 1e-4 * np.abs(ref).sum(0))
