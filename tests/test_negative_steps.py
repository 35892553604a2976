"""run_steps_any (aloha_gb300/csrc/steps.h) from negative ray parameters equals
the loop it replaces, bit for bit (tests/cpp/negative_steps_check.cpp, the header
the kernels use compiled for the host), and frames that start there equal the
oracle's."""
import os
import shutil
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_jump_equals_loop_from_negative_t(tmp_path):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("g++ not found")
    exe = str(tmp_path / "negative_steps_check")
    subprocess.run([cxx, "-O2", "-std=c++17", "-ffp-contract=off", "-I", os.path.join(ROOT, "aloha_gb300", "csrc"),
                    os.path.join(ROOT, "tests", "cpp", "negative_steps_check.cpp"), "-o", exe], check=True)
    out = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert out.returncode == 0, out.stdout + out.stderr
    assert " mismatches 0" in out.stdout


@pytest.mark.gpu
@pytest.mark.parametrize("dt,jitter", [(0.3, 462550464.0), (0.971369, 69312904.0), (0.5, 2.0**33)])
@pytest.mark.parametrize("bricks", [1, 5])
def test_frames_equal_the_oracle(gpu_ctx_factory, oracle, dt, jitter, bricks):
    from aloha_gb300 import abi
    from aloha_gb300 import scenes as S
    from aloha_gb300 import volfile as V

    dims, W, H = (40, 30, 34), 60, 44
    # empty around a small core: the march jumps from its first sample on
    vol = S.blob_field(dims, 3, (2.0, 3.0), seed=101)
    descs = S.single_brick(dims) if bricks == 1 else V.chopsuey_split(dims, bricks)
    vox = S.extract_bricks(vol, descs)
    tf = S.ramp_tf()
    cam = S.orbit_cameras(dims, 1, W, H, seed=103, distance=0.3, fovy=80.0)[0]  # the eye inside the volume
    params = dict(dt=dt, jitter_mode=abi.JITTER_CONST, jitter_value=jitter)
    ctx = gpu_ctx_factory()
    ctx.set_bricks(descs, vox)
    ctx.set_transfer_function(tf)
    ctx.set_params(**params)
    ctx.set_camera(0, *cam)
    ctx.resize(0, W, H)
    for ranks in dict.fromkeys((bricks, 1)):
        ctx.set_ranks(ranks)
        ref = oracle.render(descs, vox, tf, oracle.make_camera(*cam), W, H, oracle.make_params(**params),
                            n_ranks=ranks, want=("fb", "rank_images", "final"))
        for order in (abi.CHUNKS_RING, abi.CHUNKS_PROBED):
            ctx.set_chunk_order(order)
            np.testing.assert_array_equal(ctx.render(0, width=W, height=H), ref["fb"])
            assert ctx.stats().samples == ref["samples"]
            images = np.zeros((ranks, H, W, 4), np.float32)
            ctx.render_partials(0, images)
            np.testing.assert_array_equal(images, ref["rank_images"])
    # the training forward, and its replay over the empty macrocells
    img = np.zeros((H, W, 4), np.float32)
    ctx.forward(0, img, 32)
    np.testing.assert_array_equal(img, ref["final"])
    samples = ctx.stats().samples
    ctx.backward(0, np.ones((H, W, 4), np.float32), None, np.zeros(dims[::-1], np.float32), (0, 0, 0), dims)
    assert ctx.stats().samples == samples
