"""The standalone composite takes device images without allocating or waiting,
with its order in the launch parameters up to 1024 ranks; beyond that, and for
host buffers, through device scratch.  All give the same frame."""
import numpy as np
import pytest

from aloha_gb300 import abi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ranks", [1, 2, 1023, 1024, 1025])
@pytest.mark.parametrize("mode", [abi.COMPOSITE_FP32, abi.COMPOSITE_UBYTE])
def test_device_and_host_images_agree(gpu_ctx_factory, ranks, mode):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(ranks)
    W, H = 13, 7
    a = rng.random((ranks, H, W, 1), dtype=np.float32) * np.float32(0.02)
    img = np.concatenate([rng.random((ranks, H, W, 3), dtype=np.float32) * a, a], axis=3)
    q = rng.integers(0, 1 << 24, (ranks, H, W)).astype(np.uint32) | np.uint32(3 << 24)
    order = rng.permutation(ranks).astype(np.int32)
    host = abi.composite_over(img, order, W, H, mode)
    host8 = abi.composite_over_rgba8(q, order, W, H)
    dev = torch.from_numpy(img).cuda()
    dev8 = torch.from_numpy(q.view(np.int32)).cuda()
    for stream in (None, torch.cuda.current_stream(), torch.cuda.Stream()):
        fb = torch.zeros((H, W), dtype=torch.int32, device="cuda")
        fb8 = torch.zeros_like(fb)
        torch.cuda.synchronize()
        abi.composite_over(dev, order, W, H, mode, fb, stream)
        abi.composite_over_rgba8(dev8, order, W, H, fb8, stream)
        torch.cuda.synchronize()
        np.testing.assert_array_equal(fb.cpu().numpy().view(np.uint32), host)
        np.testing.assert_array_equal(fb8.cpu().numpy().view(np.uint32), host8)
    for bad in (np.append(order[:-1], ranks), np.append(order[:-1], -1)):
        with pytest.raises(abi.AlohaError) as e:
            abi.composite_over(dev, bad, W, H, mode, fb)
        assert e.value.code == abi.ERR_OUT_OF_RANGE
