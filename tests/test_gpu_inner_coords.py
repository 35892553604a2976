"""Scenes on both sides of every bound of the unclamped coordinates
(InnerCoords in aloha_gb300/csrc/internal.h): frames and sample counts equal
the oracle's, also when a bound is crossed between replays of a graph."""
import numpy as np
import pytest

from aloha_gb300 import abi
from aloha_gb300 import scenes as S
from aloha_gb300 import volfile as V

pytestmark = pytest.mark.gpu

W, H = 50, 38


def shifted(descs, by, grow=0.0):
    out = []
    for d in descs:
        d = {k: list(v) for k, v in d.items()}
        for key in ("cell_lo", "cell_hi", "voxel_lo", "voxel_hi", "space_lo", "space_hi"):
            d[key] = [v + by for v in d[key]]
        d["space_lo"] = [v - grow for v in d["space_lo"]]
        d["space_hi"] = [v + grow for v in d["space_hi"]]
        out.append(d)
    return out


def volume(dims, peak=1.0, low=0.0):
    vol = S.blob_field(dims, 6, (2.0, 5.0), seed=67)
    vol[dims[2] // 2, dims[1] // 2, dims[0] // 2] = peak
    vol[0, 0, 0] = low
    return vol


CASES = {
    "plain": {},
    "largest values": dict(peak=1024.0, low=-1024.0),
    "wide values": dict(peak=1500.0),
    "wide negative": dict(low=-4096.0),
    "near eye bound": dict(distance=1300.0, fovy=0.05),
    "far eye": dict(distance=2000.0, fovy=0.03),
    "box beyond its voxels": dict(grow=3.0),
    "brick near the space bound": dict(shift=16340),
    "brick past the space bound": dict(shift=16380),
    "large steps": dict(dt=1000.0, jitter_mode=abi.JITTER_NONE),
    "larger steps": dict(dt=1500.0, jitter_mode=abi.JITTER_NONE),
    "jitter bound": dict(jitter_mode=abi.JITTER_CONST, jitter_value=-16.0),
    "large jitter": dict(jitter_mode=abi.JITTER_CONST, jitter_value=17.25),
    "flat camera": dict(flat=True),
    "one voxel thick": dict(dims=(24, 24, 1)),
    "largest table": dict(tf_n=2048, peak=1024.0),
    "inside": dict(distance=0.2, fovy=80.0),
}


@pytest.mark.parametrize("name", CASES)
@pytest.mark.parametrize("bricks", [1, 6])
def test_frames_equal_the_oracle(gpu_ctx_factory, oracle, name, bricks):
    c = CASES[name]
    dims = c.get("dims", (26, 22, 24))
    vol = volume(dims, c.get("peak", 1.0), c.get("low", 0.0))
    descs = S.single_brick(dims) if bricks == 1 else V.chopsuey_split(dims, bricks)
    vox = S.extract_bricks(vol, descs)
    descs = shifted(descs, c.get("shift", 0), c.get("grow", 0.0))
    tf = S.ramp_tf(c.get("tf_n", 256))
    cam = S.orbit_cameras(dims, 1, W, H, seed=71, distance=c.get("distance", 1.5), fovy=c.get("fovy", 45.0))[0]
    org = (np.asarray(cam[0], np.float64) + c.get("shift", 0)).astype(np.float32)
    cam = (org,) + tuple(cam[1:])
    if c.get("flat"):
        cam = (cam[0], np.asarray(cam[1]) + 25 * np.asarray(cam[2]), np.zeros(3, np.float32), cam[3])
    params = {k: c[k] for k in ("dt", "jitter_mode", "jitter_value") if k in c}
    ctx = gpu_ctx_factory()
    ctx.set_bricks(descs, vox)
    ctx.set_transfer_function(tf)
    ctx.set_params(**params)
    ctx.set_camera(0, *cam)
    ctx.resize(0, W, H)
    ref = oracle.render(descs, vox, tf, oracle.make_camera(*cam), W, H, oracle.make_params(**params), n_ranks=len(descs))
    np.testing.assert_array_equal(ctx.render(0, width=W, height=H), ref["fb"])
    assert ctx.stats().samples == ref["samples"]
    one = oracle.render(descs, vox, tf, oracle.make_camera(*cam), W, H, oracle.make_params(**params), n_ranks=1,
                        want=("final",))
    ctx.set_ranks(1)
    img = np.zeros((H, W, 4), np.float32)
    ctx.forward(0, img, 32)
    np.testing.assert_array_equal(img, one["final"])


def test_bounds_crossed_between_graph_replays(gpu_ctx_factory, oracle):
    torch = pytest.importorskip("torch")
    dims = (26, 22, 24)
    descs = V.chopsuey_split(dims, 4)
    plain, wide = volume(dims), volume(dims, peak=3000.0)
    tf = S.ramp_tf()
    near = S.orbit_cameras(dims, 1, W, H, seed=73, distance=1.5)[0]
    far = S.orbit_cameras(dims, 1, W, H, seed=73, distance=2000.0, fovy=0.03)[0]
    ctx = gpu_ctx_factory()
    ctx.set_bricks(descs, S.extract_bricks(plain, descs))
    ctx.set_transfer_function(tf)
    ctx.set_params()
    ctx.set_camera(0, *near)
    ctx.resize(0, W, H)
    fb = torch.zeros((H, W), dtype=torch.int32, device="cuda")
    batch = ctx.batch([0], [fb])
    batch.launch()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        batch.launch(torch.cuda.current_stream())
    for vol, cam in ((plain, near), (wide, near), (plain, far), (wide, far), (plain, near)):
        vox = S.extract_bricks(vol, descs)
        for b, v in enumerate(vox):
            ctx.update_brick(b, v)
        ctx.set_camera(0, *cam)
        ref = oracle.render(descs, vox, tf, oracle.make_camera(*cam), W, H, oracle.make_params(), n_ranks=len(descs))
        assert ctx.composite_order(0)  # brings the view's device state up to date
        for replay in (graph.replay, batch.launch_graph):
            fb.zero_()
            torch.cuda.synchronize()
            replay()
            torch.cuda.synchronize()
            np.testing.assert_array_equal(fb.cpu().numpy().view(np.uint32), ref["fb"])
    batch.close()
