"""Frames rendered with two lanes per ray: ragged and tiny frames in ring order,
the largest frame in ring order that takes this path next to the smallest that
does not, and cost-ordered frames whose counts choose it (or, for short rays or
early ends, may not), over odd and even sample counts per brick, several passes,
ranks, and the output stage's options.  Frames, rank images, depths and sample
counts must equal the oracle's."""
import numpy as np
import pytest

from aloha_gb300 import abi
from aloha_gb300 import scenes as S
from aloha_gb300 import volfile as V

pytestmark = pytest.mark.gpu

OPTIONS = [dict(), dict(dt=0.3), dict(dt=1.0, jitter_mode=abi.JITTER_NONE), dict(dt=40.0), dict(spp=3, crosshair=1),
           dict(et_alpha=0.3), dict(heat_map=1, heat_map_scale=0.02, composite_mode=abi.COMPOSITE_UBYTE)]


def scene(dims, bricks):
    vol = S.blob_field(dims, 12, (min(dims) / 14, min(dims) / 6), seed=sum(dims))
    descs = S.single_brick(dims) if bricks == 1 else V.chopsuey_split(dims, bricks)
    return descs, S.extract_bricks(np.asarray(vol), descs), S.ramp_tf()


def context(make, descs, vox, tf, ranks, kw):
    ctx = make()
    ctx.set_bricks(descs, vox)
    ctx.set_transfer_function(tf)
    ctx.set_ranks(ranks)
    ctx.set_params(**kw)
    return ctx


@pytest.mark.parametrize("kw", OPTIONS)
@pytest.mark.parametrize("dims,bricks,ranks,size,chunks", [
    ((48, 40, 56), 1, 1, (1, 1), abi.CHUNKS_RING), ((48, 40, 56), 5, 1, (5, 3), abi.CHUNKS_RING),
    ((48, 40, 56), 5, 5, (70, 43), abi.CHUNKS_AUTO), ((9, 130, 7), 3, 2, (61, 90), abi.CHUNKS_RING),
    ((48, 40, 56), 5, 5, (70, 43), abi.CHUNKS_PROBED), ((100, 90, 120), 1, 1, (131, 94), abi.CHUNKS_PROBED),
    ((6, 5, 7), 1, 1, (90, 66), abi.CHUNKS_PROBED)])
def test_pairs_equal_oracle(gpu_ctx_factory, oracle, dims, bricks, ranks, size, chunks, kw):
    descs, vox, tf = scene(dims, bricks)
    W, H = size
    ctx = context(gpu_ctx_factory, descs, vox, tf, ranks, kw)
    ctx.set_chunk_order(chunks)
    for cam in S.orbit_cameras(dims, 2, W, H, seed=91, distance=1.3):
        ctx.set_camera(0, *cam)
        ctx.resize(0, W, H)
        ref = oracle.render(descs, vox, tf, oracle.make_camera(*cam), W, H, oracle.make_params(**kw), n_ranks=ranks,
                            want=("fb", "rank_images", "rank_depth"))
        np.testing.assert_array_equal(ctx.render(0, width=W, height=H), ref["fb"])
        assert ctx.stats().samples == ref["samples"]
        imgs = np.zeros((ranks, H, W, 4), np.float32)
        depth = np.zeros((ranks, H, W), np.float32)
        ctx.render_partials(0, imgs, depth)
        np.testing.assert_array_equal(imgs, ref["rank_images"])
        np.testing.assert_array_equal(depth, ref["rank_depth"])


@pytest.mark.parametrize("size", [(16384, 16), (16384, 17)])
def test_ring_order_limit(gpu_ctx_factory, oracle, size):
    dims = (24, 20, 28)
    descs, vox, tf = scene(dims, 2)
    W, H = size
    ctx = context(gpu_ctx_factory, descs, vox, tf, 2, {})
    ctx.set_chunk_order(abi.CHUNKS_RING)
    cam = S.orbit_cameras(dims, 1, W, H, seed=92, distance=1.3)[0]
    ctx.set_camera(0, *cam)
    ctx.resize(0, W, H)
    ref = oracle.render(descs, vox, tf, oracle.make_camera(*cam), W, H, oracle.make_params(), n_ranks=2)
    np.testing.assert_array_equal(ctx.render(0, width=W, height=H), ref["fb"])
    assert ctx.stats().samples == ref["samples"]
