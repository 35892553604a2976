"""Scene changes with device-resident voxels, then a frame at once on a stream
that does not wait for the default one: the frame is the new scene's."""
import numpy as np
import pytest

from aloha_gb300 import scenes as S

pytestmark = pytest.mark.gpu

DIMS, W, H = (26, 22, 24), 50, 38


def volume(seed, peak=None):
    vol = S.blob_field(DIMS, 6, (2.0, 5.0), seed=seed)
    if peak is not None:
        vol[12, 11, 13] = peak
    return vol


@pytest.fixture
def scene(gpu_ctx_factory, oracle):
    torch = pytest.importorskip("torch")
    ctx = gpu_ctx_factory()
    cam = S.orbit_cameras(DIMS, 1, W, H, seed=79, distance=1.5)[0]
    plain = S.single_brick(DIMS)
    tf = S.ramp_tf()
    ctx.set_bricks(plain, [torch.from_numpy(volume(83)).cuda()])
    ctx.set_transfer_function(tf)
    ctx.set_params()
    ctx.set_camera(0, *cam)
    ctx.resize(0, W, H)
    side = torch.cuda.Stream()
    fb = torch.zeros((H, W), dtype=torch.int32, device="cuda")

    def expect(descs, vol, table):
        ctx.render(0, fb, stream=side)
        side.synchronize()
        want = oracle.render(descs, [np.ascontiguousarray(vol)], table, oracle.make_camera(*cam), W, H,
                             oracle.make_params(), n_ranks=1)
        np.testing.assert_array_equal(fb.cpu().numpy().view(np.uint32), want["fb"])

    expect(plain, volume(83), tf)
    return ctx, torch, plain, tf, expect


def test_bricks_that_change_the_form_of_the_march(scene):
    """A box beyond its voxels, values beyond the unclamped lookup's, and back."""
    ctx, torch, plain, tf, expect = scene
    beyond = [dict(plain[0], space_lo=[-1.0, 0.0, 0.0], space_hi=[DIMS[0] + 1.0, *map(float, DIMS[1:])])]
    for k in range(3):
        vol, wide = volume(89 + k), volume(97 + k, peak=3000.0)
        dev, dev_wide = torch.from_numpy(vol).cuda(), torch.from_numpy(wide).cuda()
        ctx.set_bricks(beyond, [dev])
        expect(beyond, vol, tf)
        ctx.set_bricks(plain, [dev])
        expect(plain, vol, tf)
        ctx.update_brick(0, dev_wide)
        expect(plain, wide, tf)
        ctx.update_brick(0, dev)
        expect(plain, vol, tf)


def test_tables(scene):
    ctx, torch, plain, tf, expect = scene
    vol = volume(83)
    for n in (16, 2048, 100, 256):
        table = S.seeded_tf(n, n)
        ctx.set_transfer_function(table)
        expect(plain, vol, table)
