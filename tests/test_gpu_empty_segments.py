"""The training forward sorts K-sample segments into those with a sample
outside empty macrocells and all-empty ones, which the backward treats apart
(nothing but the transfer function's alpha entries gets gradient there).  The
edges of that split: more segments per ray than the forward tracks, rays with
only one kind of segment, segments that cross bricks, the smallest and largest
transfer function, one view per launch and several."""
import numpy as np
import pytest

from aloha_gb300 import abi
from aloha_gb300 import scenes as S
from aloha_gb300 import volfile as V
from tests import scenes_for_tests as T

pytestmark = pytest.mark.gpu

CASES = [
    dict(k=1, bricks=1),                       # over 64 segments per ray
    dict(k=2, bricks=8),                       # between 32 and 64, and over
    dict(k=5, bricks=8, dt=0.3),               # inexact steps, segments across bricks
    dict(k=32, bricks=1, alpha="zero"),        # every segment empty
    dict(k=32, bricks=8, alpha="all"),         # none empty
    dict(k=16, bricks=1, n_tf=2),
    dict(k=64, bricks=8, n_tf=2048),
    dict(k=700, bricks=1, jitter_mode=abi.JITTER_NONE),  # one segment per ray
]


@pytest.mark.parametrize("case", CASES)
def test_gradients_and_sample_counts(gpu_ctx_factory, oracle, case):
    n, W, H = 40, 56, 44
    dims = (n, n - 3, n + 2)
    vol = S.blob_field(dims, 8, (2.0, 5.0), seed=53)
    descs = S.single_brick(dims) if case["bricks"] == 1 else V.chopsuey_split(dims, case["bricks"])
    vox = S.extract_bricks(vol, descs)
    tf = S.ramp_tf(case.get("n_tf", 256))
    if case.get("alpha") == "zero":
        tf[:, 3] = 0.0
    elif case.get("alpha") == "all":
        tf[:, 3] = 0.01 + 0.2 * tf[:, 3]
    params = {k: case[k] for k in ("dt", "jitter_mode") if k in case}
    ctx = gpu_ctx_factory()
    ctx.set_bricks(descs, vox)
    ctx.set_transfer_function(tf)
    ctx.set_ranks(1)
    ctx.set_params(**params)
    cams = T.cameras(dims, 3, W, H, seed=59)
    rng = np.random.default_rng(61)
    dls = [rng.uniform(-1, 1, (H, W, 4)).astype(np.float32) for _ in cams]
    for v, cam in enumerate(cams):
        ctx.set_camera(v, *cam)
        ctx.resize(v, W, H)
    ctx.forward_views([0, 1, 2], [np.zeros((H, W, 4), np.float32) for _ in cams], case["k"])
    samples = ctx.stats().samples
    ref_tf, ref_den = np.zeros((tf.shape[0], 4)), np.zeros(dims[::-1])
    for cam, dl in zip(cams, dls):
        r = oracle.adjoint(descs, vox, tf, oracle.make_camera(*cam), W, H, dl, (0, 0, 0), dims,
                           oracle.make_params(**params))
        ref_tf += r["dtf"]
        ref_den += r["ddensity"]

    def check(got, ref):
        scale = np.linalg.norm(ref)
        assert np.linalg.norm(got - ref) <= 5e-4 * scale

    for want_tf, want_den in ((True, True), (True, False), (False, True)):
        grid = ((0, 0, 0), dims) if want_den else (None, None)
        for together in (True, False):  # one launch for all views, and one call per view
            dtf = np.zeros((tf.shape[0], 4), np.float32) if want_tf else None
            dden = np.zeros(dims[::-1], np.float32) if want_den else None
            total = 0
            for views in ([[0, 1, 2]] if together else [[0], [1], [2]]):
                ctx.backward_views(views, [dls[v] for v in views], dtf, dden, *grid)
                total += ctx.stats().samples
            assert total == samples
            if want_tf:
                check(dtf, ref_tf)
            if want_den:
                check(dden, ref_den)
