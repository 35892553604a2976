"""The composite's device buffers after its asynchronous call: the binding keeps
them from other work until the kernel is done, whichever stream they were
allocated on."""
import numpy as np
import pytest

from aloha_gb300 import abi

torch = pytest.importorskip("torch")


class Stream:
    def __init__(self, ptr, log):
        self.cuda_stream, self.log = ptr, log

    def synchronize(self):
        self.log.append(("wait", self.cuda_stream))


def device_like(log, name):
    class T(torch.Tensor):
        is_cuda = property(lambda self: True)

        def record_stream(self, stream):
            log.append((name, stream.cuda_stream))

    return torch.Tensor._make_subclass(T, torch.zeros(4))


class Raw:
    """Device memory of another library."""

    def data_ptr(self):
        return 16

    def is_contiguous(self):
        return True


@pytest.mark.parametrize("call", [abi.composite_over, abi.composite_over_rgba8])
def test_buffers_are_held_until_the_kernel_is_done(monkeypatch, call):
    log = []

    class Lib:
        def aloha_composite_over(self, *a):
            return abi.OK

        aloha_composite_over_rgba8 = aloha_composite_over

    monkeypatch.setattr(abi, "lib", lambda: Lib())
    monkeypatch.setattr(torch.cuda, "current_stream", lambda *a: Stream(64, log))
    monkeypatch.setattr(torch.cuda, "ExternalStream", lambda ptr: Stream(ptr, log))
    images, fb = device_like(log, "images"), device_like(log, "fb")
    order = np.zeros(1, np.int32)
    run = lambda images, fb, stream: call(images, order, 2, 2, fb=fb, stream=stream)
    run(images, fb, Stream(64, log))
    assert sorted(log) == [("fb", 64), ("images", 64)]
    log.clear()
    run(images, fb, Stream(128, log))  # not the current stream
    assert log == [("wait", 128)]
    log.clear()
    run(Raw(), fb, Stream(64, log))  # nothing to record the stream on
    assert log == [("wait", 64)]
    log.clear()
    run(np.zeros((1, 2, 2, 4), np.float32), np.zeros((2, 2), np.uint32), None)  # host memory: the call has waited
    assert log == []


@pytest.mark.gpu
@pytest.mark.parametrize("fmt", ["f32", "rgba8"])
@pytest.mark.parametrize("where", ["default", "side"])
def test_images_of_another_stream_dropped_after_the_call(fmt, where):
    n, w, h = 16, 640, 360
    rng = np.random.default_rng(3)
    order = rng.permutation(n).astype(np.int32)
    if fmt == "f32":
        host = rng.random((n, h, w, 4), np.float32)
        host[..., :3] *= host[..., 3:]
        want = abi.composite_over(host, order, w, h)
    else:
        host = rng.integers(0, 2**31, (n, h, w)).astype(np.int32)
        want = abi.composite_over_rgba8(host.view(np.uint32), order, w, h)
    owner = torch.cuda.Stream()
    run = torch.cuda.default_stream() if where == "default" else torch.cuda.Stream()
    busy = torch.rand((4096, 4096), device="cuda")
    for _ in range(4):
        fb = torch.zeros((h, w), dtype=torch.int32, device="cuda")
        with torch.cuda.stream(owner):
            images = torch.from_numpy(host).cuda()
        torch.cuda.synchronize()
        with torch.cuda.stream(run):
            for _ in range(8):
                busy = busy @ busy / 4096.0  # the composite waits behind this
            if fmt == "f32":
                abi.composite_over(images, order, w, h, fb=fb, stream=run)
            else:
                abi.composite_over_rgba8(images, order, w, h, fb=fb, stream=run)
        shape, dtype = images.shape, images.dtype
        del images
        with torch.cuda.stream(owner):
            torch.full(shape, 7, dtype=dtype, device="cuda")  # the same memory, unless it is held
        torch.cuda.synchronize()
        np.testing.assert_array_equal(fb.cpu().numpy().view(np.uint32), want)


@pytest.mark.gpu
def test_parameters_that_require_grad(gpu_ctx_factory):
    images = torch.rand((2, 8, 8, 4), device="cuda").requires_grad_()
    fb = torch.zeros((8, 8), dtype=torch.int32, device="cuda")
    abi.composite_over(images, np.array([1, 0], np.int32), 8, 8, fb=fb, stream=torch.cuda.current_stream())
    want = abi.composite_over(images.detach().cpu().numpy(), np.array([1, 0], np.int32), 8, 8)
    np.testing.assert_array_equal(fb.cpu().numpy().view(np.uint32), want)
