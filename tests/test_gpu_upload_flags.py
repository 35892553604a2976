"""The upload's flags: a voxel that is not finite is found wherever it lies, and
values beyond the unclamped march's range cost an upload next to nothing."""
import time

import numpy as np
import pytest

from aloha_gb300 import abi
from aloha_gb300 import scenes as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
@pytest.mark.parametrize("wide", [False, True])
def test_a_single_bad_voxel_is_found(gpu_ctx_factory, bad, wide):
    nx, ny, nz = 130, 9, 6  # two chunks of columns, rows and slices beyond a macrocell
    plain = np.full((nz, ny, nx), 5000.0 if wide else 0.5, np.float32)
    ctx = gpu_ctx_factory()
    for x in (0, 3, 4, 119, 120, 123, 124, 127, 129):
        for y, z in ((0, 0), (ny - 1, nz - 1), (4, 3), (3, 4)):
            vol = plain.copy()
            vol[z, y, x] = bad
            with pytest.raises(abi.AlohaError) as e:
                ctx.set_bricks(S.single_brick((nx, ny, nz)), [vol])
            assert e.value.code == abi.ERR_INVALID_ARGUMENT
    ctx.set_bricks(S.single_brick((nx, ny, nz)), [plain])


def test_wide_values_upload_as_fast_as_others(gpu_ctx_factory):
    """The same bytes; a CTA adds a barrier, a reduction and one read over the host
    link, which the others hide: at most 1.3 times the time."""
    torch = pytest.importorskip("torch")
    dims = (256, 256, 256)
    plain = torch.rand(dims, device="cuda")
    wide = (plain * 40000.0 - 1000.0).contiguous()
    ctx = gpu_ctx_factory()
    ctx.set_bricks(S.single_brick(dims), [plain])

    def best(v):
        times = []
        for _ in range(25):
            torch.cuda.synchronize()
            t = time.perf_counter()
            ctx.update_brick(0, v)
            times.append(time.perf_counter() - t)
        return min(times)

    best(plain)
    assert best(wide) <= 1.3 * best(plain)
