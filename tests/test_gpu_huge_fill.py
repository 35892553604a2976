"""A fill value of the type's largest magnitude next to ordinary voxels: samples
in the fill's empty macrocells leave the colour alone, wherever a run of the march
ends, so the frame is that of a harmless fill."""
import numpy as np
import pytest

from aloha_gb300 import abi
from aloha_gb300 import scenes as S

pytestmark = pytest.mark.gpu

DIMS, W, H = (8, 8, 32), 40, 24


def volume(fill):
    v = np.full(DIMS[::-1], fill, np.float32)
    v[:8] = 0.5 + 0.3 * np.random.default_rng(5).random((8, 8, 8), np.float32)
    return v


def frames(ctx, torch, fill):
    """The same frame through each form of the march.  Along z the samples of dt 2.2
    lie at 2.0, 4.2, 6.4 (their taps among the ordinary voxels 0..7) and 8.6 (in
    the fill), shifted by less than 0.1 towards the edges."""
    ctx.set_bricks(S.single_brick(DIMS), [volume(fill)])
    out = []

    def add(fb):
        torch.cuda.synchronize()
        out.append(np.asarray(fb.cpu() if hasattr(fb, "cpu") else fb).view(np.uint32).copy())

    for order in (abi.CHUNKS_RING, abi.CHUNKS_PROBED):
        ctx.set_chunk_order(order)
        add(ctx.render(0, width=W, height=H))
        assert ctx.stats().samples > 4 * W * H
    ctx.set_chunk_order(abi.CHUNKS_AUTO)
    for tile in ((8, 8), (0, 0)):
        ctx.set_render_tile(*tile)
        add(ctx.render(0, width=W, height=H))
    for staging in (abi.STAGING_NEXT_SAMPLE, abi.STAGING_NONE):
        ctx.set_render_staging(staging)
        add(ctx.render(0, width=W, height=H))
    fb = torch.zeros((H, W), dtype=torch.int32, device="cuda")
    for unroll in (1, 2):
        batch = ctx.batch([0], [fb])
        batch.set_unroll(unroll)
        batch.launch()
        add(fb)
        batch.close()
    img = np.zeros((H, W, 4), np.float32)
    ctx.forward(0, img, 4)
    out.append(img)
    return out


@pytest.mark.parametrize("fill", [3.4e38, -3.4028235e38, 1e37])
def test_frames_equal_those_of_a_harmless_fill(gpu_ctx_factory, fill):
    torch = pytest.importorskip("torch")
    ctx = gpu_ctx_factory()
    ctx.set_bricks(S.single_brick(DIMS), [volume(0.0)])
    ctx.set_transfer_function(S.ramp_tf())
    ctx.set_params(dt=2.2, jitter_mode=abi.JITTER_NONE)
    ctx.set_camera(0, np.float32([4, 4, -15.6]), np.float32([-0.06, -0.06, 1]), np.float32([0.12 / W, 0, 0]),
                   np.float32([0, 0.12 / H, 0]))
    ctx.resize(0, W, H)
    want = frames(ctx, torch, 900.0 if fill > 0 else -900.0)
    got = frames(ctx, torch, fill)
    assert (want[0] != 0).all() and np.isfinite(want[-1]).all()
    for g, w in zip(got, want):
        np.testing.assert_array_equal(g, w)


@pytest.mark.parametrize("big", [1e17, 3e38])
def test_table_of_huge_colours(gpu_ctx_factory, oracle, big):
    """Entries whose differences overflow: the lookup between them is not finite,
    but samples in empty macrocells still leave the colour alone."""
    torch = pytest.importorskip("torch")
    tf = np.zeros((64, 4), np.float32)
    tf[20:44] = S.ramp_tf(64)[20:44] + 0.1
    tf[50:, 0] = big * np.where(np.arange(14) % 2, 1, -1)  # alpha 0
    ctx = gpu_ctx_factory()
    vol = volume(0.9)
    vol[:8] = 0.45
    descs = S.single_brick(DIMS)
    ctx.set_bricks(descs, [vol])
    ctx.set_params(dt=2.2, jitter_mode=abi.JITTER_NONE)
    ctx.set_camera(0, np.float32([4, 4, -15.6]), np.float32([-0.06, -0.06, 1]), np.float32([0.12 / W, 0, 0]),
                   np.float32([0, 0.12 / H, 0]))
    ctx.resize(0, W, H)
    plain = tf.copy()
    plain[50:, 0] = 0.0
    images = []
    for table in (plain, tf, plain):
        ctx.set_transfer_function(table)
        img = np.zeros((H, W, 4), np.float32)
        ctx.forward(0, img, 4)
        images.append(img)
        images.append(ctx.render(0, width=W, height=H))
    assert np.isfinite(images[0]).all() and (images[1] != 0).all()
    for a, b in zip(images[2:], images[:2] * 2):
        np.testing.assert_array_equal(a, b)
