"""CPU model of the brick element (V(x,y,z), V(x,y,z+1), V(x,y+1,z),
V(x,y+1,z+1)), of the stencil's seven loads and of the unclamped coordinates
(aloha_gb300/csrc/march.cuh stencil, inner_axis): for coordinates across the
brick and its margin of a quarter voxel, the unclamped form addresses the same
elements with the same weights as the clamped one, all inside the padded array;
and the loads hold the clamped voxels of the 20-voxel cross for coordinates far
outside as well."""
import numpy as np
import pytest

from tests.test_layout_model import axis, clamped

APRON = 2
F = np.float32
MAGIC, MAGIC_BITS = F(12582912.0), 0x4B400000


def pitches(nx, ny):
    px = nx + 2 * APRON
    px += (2 - px) & 3
    sz = px * (ny + 2 * APRON)
    return px, sz + ((4 - sz) & 7)


def pad(vol):
    nz, ny, nx = vol.shape
    px, sz = pitches(nx, ny)
    out = np.full((sz * (nz + 2 * APRON), 4), np.nan, np.float32)
    for z in range(nz + 2 * APRON):
        for y in range(ny + 2 * APRON):
            for x in range(px):
                at = z * sz + y * px + x
                for k, (dy, dz) in enumerate(((0, 0), (0, 1), (1, 0), (1, 1))):
                    out[at, k] = clamped(vol, x - APRON, y + dy - APRON, z + dz - APRON)
    return out, px, sz


def inner_axis(u):
    """(bits, f, g, h) with the addition rounded down."""
    u = F(u)
    m = F(u - F(0.5))
    r = F(np.floor(float(u)) + float(MAGIC))  # exact in float64: the sum rounded down
    fc = F(r - MAGIC)
    d = F(m - fc)
    h = bool(d < 0)
    return int(r.view(np.uint32)), (F(d + F(1)) if h else d), F(u - fc), h


def weights(u):
    m = F(F(u) - F(0.5))
    return F(m - np.floor(m)), F(F(u) - np.floor(F(u)))


@pytest.mark.parametrize("dims", [(5, 3, 4), (1, 1, 1), (2, 7, 1), (9, 8, 10), (128, 4, 3)])
def test_unclamped_form_equals_the_clamped_one(dims):
    nx, ny, nz = dims
    rng = np.random.default_rng(sum(dims))
    vol = rng.random((nz, ny, nx), dtype=np.float32)
    q, sy, sz = pad(vol)
    assert sy % 8 in (2, 6) and sz % 8 == 4
    edge = [-0.25, -1e-7, 0.0, 1e-7, 0.25, 0.5, 0.75]

    def spread(n):
        return edge + [n - 0.5, F(n) - F(1e-6) * n, n, n + 0.25]

    inside = [(x, y, z) for x in spread(nx) for y in spread(ny)[::2] for z in spread(nz)[1::2]]
    inside += [tuple(rng.uniform(-0.25, np.array(dims) + 0.25)) for _ in range(300)]
    outside = [tuple(rng.uniform(-6, np.array(dims) + 6)) for _ in range(200)] + [(-1e9, 1e9, 0.5), (3e38, -3e38, 1e30)]
    origin = (APRON * sz + APRON * sy + APRON)
    inner_origin = (-MAGIC_BITS * (1 + sy + sz)) & 0xFFFFFFFF
    for k, u in enumerate(inside + outside):
        i, c, h = zip(*(axis(v, n, False) for v, n in zip(u, dims)))
        e = [ii if hh else ii + 2 for ii, hh in zip(i, h)]
        at = c[2] * sz + c[1] * sy + c[0]
        offs = [e[0] - c[0], (e[1] - c[1]) * sy, (e[2] - c[2]) * sz]
        if k < len(inside):
            b, f, g, hh = zip(*(inner_axis(v) for v in u))
            at32 = (b[2] * sz + inner_origin + b[1] * sy + b[0]) & 0xFFFFFFFF
            assert (at32 - (1 << 32) if at32 >> 31 else at32) == at
            assert [(-1 if x else 2) * s for x, s in zip(hh, (1, sy, sz))] == offs and list(hh) == list(h)
            assert [(x, y) for x, y in zip(f, g)] == [weights(v) for v in u]

        def elem(offset):
            assert 0 <= origin + at + offset < len(q)
            return q[origin + at + offset]

        for col, x in ((elem(0), c[0]), (elem(1), c[0] + 1), (elem(offs[0]), e[0])):
            assert list(col) == [clamped(vol, x, c[1] + dy, c[2] + dz) for dy, dz in ((0, 0), (0, 1), (1, 0), (1, 1))]
        for dx in (0, 1):
            assert list(elem(offs[1] + dx)[:2]) == [clamped(vol, c[0] + dx, e[1], c[2] + dz) for dz in (0, 1)]
            assert list(elem(offs[2] + dx)[::2]) == [clamped(vol, c[0] + dx, c[1] + dy, e[2]) for dy in (0, 1)]
