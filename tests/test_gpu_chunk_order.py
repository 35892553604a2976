"""The cost-ordered chunk list at the edges of its sort: frames whose ring slots
fill one sort block or just more, and the largest frames that sort in two
launches next to the smallest that take three.  Each list must hold every chunk
once, again and again (its counts are zeroed by the launch that reads them):
frames of changing cameras and sizes equal those of the ring order."""
import numpy as np
import pytest

from aloha_gb300 import abi
from aloha_gb300 import scenes as S

from tests import scenes_for_tests as T

pytestmark = pytest.mark.gpu

# (width, height): 8x4 chunks; the longer side in chunks sets the ring's slots.
# 31 chunks a side: 961 slots (one sort block); 32: 1089 (two); 1061: 1100 blocks; 1063: 1104
SIZES = [(31 * 8, 90), (32 * 8, 90), (1061 * 8 - 3, 6), (1063 * 8, 5), (9, 1061 * 4), (9, 1063 * 4 - 1)]


@pytest.mark.parametrize("size", SIZES)
def test_probed_order_holds_every_chunk(gpu_ctx_factory, size):
    W, H = size
    vol, descs, vox, tf = T.chopsuey_scene(32, 8)
    ctx = gpu_ctx_factory()
    ctx.set_bricks(descs, vox)
    ctx.set_transfer_function(tf)
    ctx.set_params()
    ctx.set_render_split(abi.SPLIT_PIXELS)
    cams = S.orbit_cameras((32, 32, 32), 2, W, H, seed=83, distance=1.1)
    frames = {}
    for mode in (abi.CHUNKS_RING, abi.CHUNKS_PROBED):
        ctx.set_chunk_order(mode)
        frames[mode] = []
        for w, h in [(W, H), (W, H), (48, 40), (W, H)]:  # another size moves the table
            for cam in cams:
                ctx.set_camera(0, *cam)
                ctx.resize(0, w, h)
                frames[mode].append((np.array(ctx.render(0, width=w, height=h)), ctx.stats().samples))
    for (got, n_got), (want, n_want) in zip(frames[abi.CHUNKS_PROBED], frames[abi.CHUNKS_RING]):
        np.testing.assert_array_equal(got, want)
        assert n_got == n_want
    assert frames[abi.CHUNKS_RING][0][1] > 0
