"""Cost-ordered frames recorded into CUDA graphs among frames of other sizes: a
recording that is never replayed leaves nothing behind, and a replay after frames
of other sizes renders its own."""
import numpy as np
import pytest

from aloha_gb300 import abi
from aloha_gb300 import scenes as S

pytestmark = pytest.mark.gpu


def test_recorded_frames_among_others(gpu_ctx_factory):
    torch = pytest.importorskip("torch")
    dims = (48, 40, 44)
    descs = S.single_brick(dims)
    ctx = gpu_ctx_factory()
    ctx.set_bricks(descs, S.extract_bricks(S.blob_field(dims, 8, (4.0, 9.0), seed=127), descs))
    ctx.set_transfer_function(S.ramp_tf())
    ctx.set_params()
    sizes = [(640, 480), (96, 64), (1024, 768), (801, 603)]
    fbs, want = [], []
    ctx.set_chunk_order(abi.CHUNKS_RING)
    for v, (w, h) in enumerate(sizes):
        ctx.set_camera(v, *S.orbit_cameras(dims, 1, w, h, seed=131 + v, distance=1.3)[0])
        ctx.resize(v, w, h)
        fbs.append(torch.zeros((h, w), dtype=torch.int32, device="cuda"))
        ctx.render(v, fbs[v])
        torch.cuda.synchronize()
        want.append(fbs[v].clone())
    ctx.set_chunk_order(abi.CHUNKS_PROBED)
    side = torch.cuda.Stream()

    def check(v, launch):
        fbs[v].zero_()
        torch.cuda.synchronize()
        launch()
        torch.cuda.synchronize()
        assert torch.equal(fbs[v], want[v]), sizes[v]

    def render(v):
        check(v, lambda: ctx.render(v, fbs[v], side))

    def record(v):
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.stream(side), torch.cuda.graph(graph, stream=side):
            ctx.render(v, fbs[v], side)
        return graph

    render(2)  # the largest first: recording allocates nothing
    render(0)
    dropped = record(1)  # never replayed
    for v in (1, 1, 0, 3):
        render(v)
    graphs = [record(v) for v in range(4)]
    for v in (3, 0, 2, 1):
        check(v, graphs[v].replay)
        render((v + 1) % 4)
        check(v, graphs[v].replay)
        check(v, graphs[v].replay)
    del dropped
    assert np.count_nonzero(want[0].cpu().numpy()) > 1000
