"""Workloads of the volume path, each one pass through the public binding.

Kinds: a single frame into device or page-locked host memory (viewer,
headless), a batch of views of uneven bricks in one graph launch, per-rank
images with their composite (an external compositor), a composite of rank
images alone, a time step of a volume that changes between frames, and a
training step of the differentiable form.  Volumes are seeded Gaussian-blob
fields with a ramp transfer function and orbit cameras, at the configured
sizes and at odd ones between and around them.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from aloha_gb300 import abi
from aloha_gb300 import scenes as S
from aloha_gb300 import volfile as V
from aloha_gb300.autograd import DifferentiableRenderer, render_views

_FRAME = dict(kind="frame", bricks=1, ranks=1, dt=0.5, jitter="hash", spp=1, mode="fp32", tf_n=256, blobs=16,
              distance=2.0, fovy=45.0, host=False, crosshair=False)
_TRAIN = dict(kind="train", bricks=1, dt=0.5, jitter="hash", tf_n=256, blobs=16, distance=2.0, fovy=45.0, k=32)


def _case(base, name, dims, size, **kw):
    c = dict(base, nx=dims[0], ny=dims[1], nz=dims[2], width=size[0], height=size[1])
    c.update(kw)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # The plain configuration: a small single-brick volume, a thumbnail-sized frame; launches and host work count.
        _case(_FRAME, "frame_64", (64, 64, 64), (512, 512), blobs=8),
        # An odd-sized scan in a few bricks as one rank, rendered with oversampling, an inexact step and 8-bit
        # compositing into an odd window with the reference's crosshair.
        _case(_FRAME, "frame_odd_spp2", (181, 113, 237), (701, 395), bricks=5, dt=0.3, spp=2, mode="ubyte", tf_n=100,
              distance=1.4, crosshair=True),
        # The headline workload as a viewer runs it: camera in, frame out into page-locked host memory.
        _case(_FRAME, "frame_512_host", (512, 512, 512), (1024, 1024), bricks=8, ranks=8, blobs=64, host=True),
        # The large configuration's render: 64 bricks as 64 virtual ranks.
        _case(_FRAME, "frame_1024_64ranks", (1024, 1024, 1024), (2048, 2048), bricks=64, ranks=64, blobs=64),
        # The batched configuration: uneven 3x2x2 bricks, two view sizes, one graph launch for all views.
        _case(_FRAME, "batch_uneven", (512, 512, 512), (1024, 1024), kind="batch", blobs=64, big=16, small=8),
        # The unfused form: per-rank float images and depths, then the ordered composite, as an external
        # compositor takes them.
        _case(_FRAME, "partials_256", (256, 256, 256), (800, 600), kind="partials", bricks=8, ranks=8, blobs=32),
        # The compositor alone: float images of many ranks at full-HD.
        _case({}, "composite_f32", (0, 0, 0), (1920, 1080), kind="composite", ranks=16, fmt="f32", mode="fp32"),
        # A simulation's time step: every brick replaced, the transfer function retuned, one frame rendered.
        _case(_FRAME, "series_256", (256, 256, 256), (512, 512), kind="series", bricks=8, ranks=8, blobs=32),
        # The differentiable configuration: 16 small views of one brick, both gradients, one optimiser step's worth.
        _case(_TRAIN, "train_128_both", (128, 128, 128), (256, 256), views=16, want="both"),
        # Transfer-function design on a large fixed volume.
        _case(_TRAIN, "train_512_tf", (512, 512, 512), (1024, 1024), views=1, want="tf", bricks=8, blobs=64),
        # Density reconstruction from a few views; the transfer function is fixed.
        _case(_TRAIN, "train_256_density", (256, 256, 256), (512, 512), views=6, want="density", blobs=32),
        # Both gradients of a large volume in bricks, the adjoint's headline size.
        _case(_TRAIN, "train_512_both", (512, 512, 512), (1024, 1024), views=2, want="both", bricks=8, blobs=64),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    limit = max(_cost(c) for c in listed())
    while True:
        c = _draw(rng)
        if _cost(c) <= limit:
            return c


def _cost(case):
    w = work(case)
    return max(w["bytes"], w["flops"] / 50.0)


def _draw(rng):
    kind = rng.choice(["frame", "frame", "batch", "partials", "composite", "series", "train", "train"])
    if kind == "composite":
        ranks, w = _log(rng, 2, 32), _log(rng, 256, 2048)
        return _case({}, None, (0, 0, 0), (w, max(16, int(w * rng.uniform(0.4, 1.0)))), kind=kind, ranks=ranks,
                     fmt=rng.choice(["f32", "rgba8"]), mode=rng.choice(["fp32", "ubyte"]))
    top = {"frame": 640, "batch": 512, "partials": 384, "series": 384, "train": 400}[kind]
    n = _log(rng, 48, top)
    dims = tuple(max(24, int(n * rng.uniform(0.5, 1.0))) for _ in range(3))
    w = _log(rng, 160, {"frame": 1800, "batch": 900, "partials": 900, "series": 900, "train": 800}[kind])
    size = (w, max(96, int(w * rng.uniform(0.5, 1.0))))
    common = dict(tf_n=rng.choice([64, 100, 256, 256, 1024]), blobs=rng.randint(6, 64),
                  dt=rng.choice([0.5, 0.5, 0.5, 1.0, 0.3]), jitter=rng.choice(["hash", "hash", "none"]),
                  distance=round(rng.uniform(0.8, 2.5), 3), fovy=round(rng.uniform(30.0, 60.0), 2))
    if kind == "train":
        want = rng.choice(["tf", "density", "both"])
        return _case(_TRAIN, None, dims, size, views=_log(rng, 1, 4 if w > 400 else 16), want=want,
                     k=rng.choice([16, 32, 64]), bricks=rng.choice([1, 1, 4, 8]), **common)
    bricks = rng.choice([1, 2, 3, 5, 8, 12, 33, 64])
    case = _case(_FRAME, None, dims, size, kind=kind, bricks=bricks, ranks=rng.choice([1, bricks]),
                 mode=rng.choice(["fp32", "fp32", "ubyte"]), **common)
    if kind == "frame":
        case.update(spp=rng.choice([1, 1, 1, 2]), host=rng.random() < 0.4, crosshair=rng.random() < 0.2)
    elif kind == "batch":
        case.update(big=rng.randint(2, 16), small=rng.randint(1, 12))
    elif kind == "partials":
        case.update(bricks=min(bricks, 12), ranks=min(case["ranks"], 12))
    elif kind == "series":
        case.update(host=rng.random() < 0.2)
    return case


# ---------------------------------------------------------------- inputs

def _dims(case):
    return case["nx"], case["ny"], case["nz"]


def _volume(case, seed, device="cuda"):
    n = max(_dims(case))
    return S.blob_field(_dims(case), case["blobs"], (n / 16.0, n / 6.4), seed=seed, device=torch.device(device))


def _descs(case):
    dims = _dims(case)
    if case["kind"] == "batch" and dims == (512, 512, 512):
        return S.grid_split(dims, ([200, 380], [256], [300]))
    if case["bricks"] == 1:
        return S.single_brick(dims)
    return V.chopsuey_split(dims, case["bricks"])


def _cameras(case, seed, count, width, height):
    return S.orbit_cameras(_dims(case), count, width, height, seed=seed, distance=case["distance"], fovy=case["fovy"])


_JITTER = {"none": abi.JITTER_NONE, "hash": abi.JITTER_HASH}
_MODE = {"fp32": abi.COMPOSITE_FP32, "ubyte": abi.COMPOSITE_UBYTE}


def _context(case, vol):
    ctx = abi.Context(0)
    descs = _descs(case)
    ctx.set_bricks(descs, [V.brick_voxels(vol, d) for d in descs])
    if case["ranks"] == 1 and len(descs) > 1:
        ctx.set_ranks(1)
    elif case["kind"] == "partials" and len(descs) > 1:
        ctx.set_rank_assignment(list(range(len(descs))), len(descs))  # rank images in the bricks' order
    ctx.set_transfer_function(S.ramp_tf(case["tf_n"]))
    ctx.set_params(dt=case["dt"], jitter_mode=_JITTER[case["jitter"]], spp=case["spp"],
                   composite_mode=_MODE[case["mode"]], crosshair=int(case["crosshair"]))
    return ctx


def _rank_images(case, seed):
    """Premultiplied images as ranks deliver them: soft discs on an empty background."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    R, H, W = case["ranks"], case["height"], case["width"]
    c = torch.rand((R, 3), device="cuda", generator=g)
    y = torch.linspace(0, 1, H, device="cuda")[None, :, None] - (0.2 + 0.6 * c[:, 0, None, None])
    x = torch.linspace(0, 1, W, device="cuda")[None, None, :] - (0.2 + 0.6 * c[:, 1, None, None])
    a = (1.0 - (x * x + y * y) / (0.05 + 0.15 * c[:, 2, None, None])).clamp(0, 1)
    a = a * (0.5 + 0.5 * torch.rand((R, H, W), device="cuda", generator=g))
    rgb = torch.rand((R, H, W, 3), device="cuda", generator=g) * a[..., None]
    img = torch.cat([rgb, a[..., None]], dim=3).contiguous()
    if case["fmt"] == "f32":
        return img
    q = (img * 255.0 + 0.5).to(torch.int64)
    q = q[..., 0] | (q[..., 1] << 8) | (q[..., 2] << 16) | (q[..., 3] << 24)
    return torch.where(q >= 1 << 31, q - (1 << 32), q).to(torch.int32).contiguous()


def _targets(case, seed):
    """Images to fit: a soft coloured disc per view."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    H, W = case["height"], case["width"]
    y = torch.linspace(-1, 1, H, device="cuda")[None, :, None, None]
    x = torch.linspace(-1, 1, W, device="cuda")[None, None, :, None]
    col = torch.rand((case["views"], 1, 1, 4), device="cuda", generator=g)
    return (col * torch.exp(-3.0 * (x * x + y * y))).contiguous()


def prepare(case, seed):
    kind, W, H = case["kind"], case["width"], case["height"]
    st = {"kind": kind, "W": W, "H": H}
    if kind == "composite":
        st.update(images=_rank_images(case, seed), mode=_MODE[case["mode"]], fmt=case["fmt"],
                  order=np.random.default_rng(seed).permutation(case["ranks"]).astype(np.int32),
                  fb=torch.zeros((H, W), dtype=torch.int32, device="cuda"))
        return st
    if kind == "train":
        st["r"] = DifferentiableRenderer(_dims(case), bricks=_descs(case), checkpoint_every=case["k"], dt=case["dt"],
                                         jitter_mode=_JITTER[case["jitter"]])
        st["views"] = list(range(case["views"]))
        for v, cam in enumerate(_cameras(case, seed + 1, case["views"], W, H)):
            st["r"].set_camera(v, cam, W, H)
        st["tf"] = torch.from_numpy(S.ramp_tf(case["tf_n"])).cuda().requires_grad_(case["want"] != "density")
        st["density"] = _volume(case, seed).requires_grad_(case["want"] != "tf")
        # the values an optimiser writes into the parameter before the step
        st["new_density"] = st["density"].detach().clone() if case["want"] != "tf" else None
        st["target"] = _targets(case, seed)
        return st
    vol = _volume(case, seed)
    ctx = st["ctx"] = _context(case, vol)
    st["mode"] = _MODE[case["mode"]]
    if kind == "batch":
        sizes = [(W, H)] * case["big"] + [(max(8, W // 2), max(4, H // 2))] * case["small"]
        st["cams"] = [_cameras(case, seed + 1 + v, 1, w, h)[0] for v, (w, h) in enumerate(sizes)]
        for v, ((w, h), cam) in enumerate(zip(sizes, st["cams"])):
            ctx.set_camera(v, *cam)
            ctx.resize(v, w, h)
        st["fbs"] = [torch.zeros((h, w), dtype=torch.int32, device="cuda") for w, h in sizes]
        st["batch"] = ctx.batch(list(range(len(sizes))), st["fbs"])
        st["batch"].set_config(8, 4)
        return st
    st["cam"] = _cameras(case, seed + 1, 1, W, H)[0]
    ctx.set_camera(0, *st["cam"])
    ctx.resize(0, W, H)
    fb = torch.zeros((H, W), dtype=torch.int32)
    st["fb"] = fb.pin_memory() if kind == "frame" and case["host"] else fb.cuda()
    if kind == "partials":
        R = 1 if case["ranks"] == 1 else len(_descs(case))
        st["images"] = torch.zeros((R, H, W, 4), device="cuda")
        st["depth"] = torch.zeros((R, H, W), device="cuda")
    elif kind == "series":
        step = _volume(case, seed + 7)
        st["bricks"] = [V.brick_voxels(step, d) for d in _descs(case)]
        if case["host"]:
            st["bricks"] = [b.cpu().numpy() for b in st["bricks"]]
        st["tf"] = S.seeded_tf(seed, case["tf_n"])
    return st


# ------------------------------------------------------------------ a pass

def run(st):
    stream = torch.cuda.current_stream()
    kind = st["kind"]
    if kind == "composite":
        if st["fmt"] == "rgba8":
            return abi.composite_over_rgba8(st["images"], st["order"], st["W"], st["H"], st["fb"], stream)
        return abi.composite_over(st["images"], st["order"], st["W"], st["H"], st["mode"], st["fb"], stream)
    if kind == "train":
        if st["new_density"] is not None:
            with torch.no_grad():
                st["density"].copy_(st["new_density"])
        img = render_views(st["r"], st["tf"], st["density"], st["views"], (st["W"], st["H"]))
        loss = ((img - st["target"]) ** 2).sum()
        want = [t for t in (st["tf"], st["density"]) if t.requires_grad]
        return {"images": img.detach(), "grads": list(torch.autograd.grad(loss, want))}
    ctx = st["ctx"]
    if kind == "batch":
        for v, cam in enumerate(st["cams"]):
            ctx.set_camera(v, *cam)
        st["batch"].launch_graph(stream)
        return st["fbs"]
    ctx.set_camera(0, *st["cam"])
    if kind == "partials":
        ctx.render_partials(0, st["images"], st["depth"], stream)
        abi.composite_over(st["images"], ctx.composite_order(0), st["W"], st["H"], st["mode"], st["fb"], stream)
        return {"images": st["images"], "depth": st["depth"], "fb": st["fb"]}
    if kind == "series":
        for i, b in enumerate(st["bricks"]):
            ctx.update_brick(i, b)
        ctx.set_transfer_function(st["tf"])
    ctx.render(0, st["fb"], stream)
    return st["fb"]


# -------------------------------------------------------------------- work

def _samples(case, width, height):
    """Expected samples of one view: covered pixels x mean chord / dt (a cube's silhouette and chord, roughly)."""
    s = 1.0 / (2.0 * case["distance"] * math.tan(math.radians(case["fovy"]) / 2.0))
    nx, ny, nz = _dims(case)
    n = max(nx, ny, nz)
    fill = (nx * ny * nz / n ** 3) ** (2.0 / 3.0)
    covered = min(1.0, 1.2 * s * s * fill * height / width)
    chord = 0.66 * (nx * ny * nz) ** (1.0 / 3.0)
    return width * height * covered * chord / case["dt"]


_SAMPLE_FLOPS = 130.0  # 30 lerps of the stencil, the shading, the lookup and the composite
_SHARE = 0.3           # samples whose transfer-function alpha is not 0; the others contribute nothing


def work(case):
    W, H, kind = case["width"], case["height"], case["kind"]
    if kind == "composite":
        px = W * H
        return {"bytes": float(px * (case["ranks"] * (16 if case["fmt"] == "f32" else 4) + 4)),
                "flops": float(px * case["ranks"] * 8)}
    voxels = 4.0 * case["nx"] * case["ny"] * case["nz"]
    if kind == "train":
        n = case["views"] * _samples(case, W, H)
        images = case["views"] * W * H * 16.0
        # forward, and its replay with the adjoint; the transfer-function gradient needs every sample
        flops = n * _SAMPLE_FLOPS * (_SHARE + (1.0 if case["want"] != "density" else _SHARE))
        grads = voxels if case["want"] != "tf" else 0.0
        if grads:
            flops += n * _SHARE * 150.0  # 20 voxel weights and their sums
        return {"bytes": voxels + grads + 3.0 * images, "flops": flops}
    views = [(W, H)]
    if kind == "batch":
        views = [(W, H)] * case["big"] + [(W // 2, H // 2)] * case["small"]
    out = sum(4.0 * w * h for w, h in views)
    if kind == "partials":
        out += 20.0 * W * H * case["ranks"]
    flops = sum(_samples(case, w, h) for w, h in views) * case["spp"] * _SHARE * _SAMPLE_FLOPS
    return {"bytes": voxels + out, "flops": flops}


# ------------------------------------------------- the same values in 64 bits

def _hash(v):
    m = 0xFFFFFFFF
    s = (v * 747796405 + 2891336453) & m
    w = ((s >> ((s >> 28) + 4)) ^ s) * 277803737 & m
    return (w >> 22) ^ w


def _rays64(cam, W, H):
    org, d00, du, dv = (torch.tensor([float(x) for x in c], dtype=torch.float64, device="cuda") for c in cam)
    y, x = torch.meshgrid(torch.arange(H, device="cuda"), torch.arange(W, device="cuda"), indexing="ij")
    d = d00 + (x.reshape(-1, 1).double() + 0.5) * du + (y.reshape(-1, 1).double() + 0.5) * dv
    d = d / d.norm(dim=1, keepdim=True)
    return org, torch.where(d.abs() < 1e-5, torch.full_like(d, 1e-5), d)


def _slab64(org, d, desc, tmin):
    lo = (torch.tensor(desc["space_lo"], dtype=torch.float64, device="cuda") - org) / d
    hi = (torch.tensor(desc["space_hi"], dtype=torch.float64, device="cuda") - org) / d
    return torch.maximum(tmin, torch.minimum(lo, hi).amax(1)), torch.maximum(lo, hi).amin(1)


def _brick64(case, vox, desc, tf, org, d, t0, t1, ils, before):
    """Colour and transmittance after one brick of the rays (d, t0, t1) that reach it with transmittance `before`."""
    dt = case["dt"]
    first = dt * (ils + torch.floor((t0 - dt * ils) / dt))
    first = torch.where(first < t0, first + dt, first)
    steps = int(((t1 - first) / dt).max().item()) + 2
    t = first[:, None] + dt * torch.arange(steps, device="cuda", dtype=torch.float64)
    u = org + t[..., None] * d[:, None, :] - torch.tensor(desc["voxel_lo"], dtype=torch.float64, device="cuda")
    off = torch.zeros((7, 3), dtype=torch.float64, device="cuda")
    for a in range(3):
        off[1 + 2 * a, a], off[2 + 2 * a, a] = 0.5, -0.5
    n = torch.tensor(vox.shape[::-1], dtype=torch.float64, device="cuda")
    taps = (u.reshape(1, -1, 3) + off[:, None, :]) * (2.0 / (n - 1)) - 1.0
    v = torch.nn.functional.grid_sample(vox[None, None], taps[None, :, None], mode="bilinear", padding_mode="border",
                                        align_corners=True)[0, 0, :, 0].reshape(7, *t.shape)
    g = torch.stack([v[1] - v[2], v[3] - v[4], v[5] - v[6]], dim=-1)
    shade = 0.1 + 0.9 * ((g * d[:, None, :]).sum(-1) / (g + 1e-4).norm(dim=-1)).abs()
    x = v[0] * tf.shape[0] - 0.5
    i = torch.floor(x).detach()
    e = torch.cat([torch.zeros((2, 4), dtype=tf.dtype, device=tf.device), tf,
                   torch.zeros((2, 4), dtype=tf.dtype, device=tf.device)])
    at = i.clamp(-2, tf.shape[0]).long()
    c = torch.lerp(e[at + 2], e[at + 3], (x - i)[..., None])
    alpha = c[..., 3] * (t < t1[:, None])

    def transmittance(a):  # before each sample
        return before[:, None] * torch.cat([torch.ones_like(a[:, :1]), torch.cumprod(1.0 - a, dim=1)[:, :-1]], dim=1)

    with torch.no_grad():
        live = transmittance(alpha) > 1.0 - 0.99  # early termination
    alpha = alpha * live
    prior = transmittance(alpha)
    w = prior * alpha
    return ((w * shade)[..., None] * c[..., :3]).sum(1), before * torch.prod(1.0 - alpha, dim=1)


def _front_to_back(descs, org):
    """Bricks by the cells between them and the eye, a valid order for the middle-split partitions used here."""
    eye = org.tolist()
    todo = list(range(len(descs)))

    def hides(p, q):  # whether brick p can lie in front of brick q: no plane parts them with the eye on q's side
        for a in range(3):
            if descs[p]["space_lo"][a] >= descs[q]["space_hi"][a] and eye[a] <= descs[p]["space_lo"][a]:
                return False
            if descs[p]["space_hi"][a] <= descs[q]["space_lo"][a] and eye[a] >= descs[p]["space_hi"][a]:
                return False
        return True

    out = []
    while todo:
        pick = next((q for q in todo if not any(p != q and hides(p, q) and not hides(q, p) for p in todo)), todo[0])
        out.append(pick)
        todo.remove(pick)
    return out


def _march64(case, descs, leaves, tf, cam, pixels=None, chunk=6_000_000):
    """Yields (pixel indices, rgba, depth entry) of the view, some rays at a time, marched in 64 bits."""
    W, H = case["width"], case["height"]
    org, d_all = _rays64(cam, W, H)
    order = _front_to_back(descs, org)
    lo = torch.tensor([min(q["space_lo"][a] for q in descs) for a in range(3)], dtype=torch.float64, device="cuda")
    hi = torch.tensor([max(q["space_hi"][a] for q in descs) for a in range(3)], dtype=torch.float64, device="cuda")
    box = {"space_lo": lo.tolist(), "space_hi": hi.tolist()}
    zero = torch.zeros(d_all.shape[0], dtype=torch.float64, device="cuda")
    b0, b1 = _slab64(org, d_all, box, zero)
    inside = torch.nonzero(b0 < b1).reshape(-1)
    per = max(256, int(chunk / (float((hi - lo).norm()) / case["dt"])))
    for at in range(0, inside.numel(), per):
        px = inside[at:at + per]
        d = d_all[px]
        rgb = torch.zeros((px.numel(), 3), dtype=torch.float64, device="cuda")
        trans = torch.ones(px.numel(), dtype=torch.float64, device="cuda")
        tmin = torch.zeros_like(trans)
        near = torch.full_like(trans, math.inf)
        draws = torch.zeros(px.numel(), dtype=torch.int64, device="cuda")
        for b in order:
            t0, t1 = _slab64(org, d, descs[b], tmin)
            hit = (t0 < t1) & (trans.detach() > 1.0 - 0.99)
            at_b = torch.nonzero(hit).reshape(-1)
            if not at_b.numel():
                continue
            ils = torch.zeros(at_b.numel(), dtype=torch.float64, device="cuda")
            if case["jitter"] == "hash":
                h = _hash(px[at_b] ^ _hash(0 ^ _hash(draws[at_b])))
                ils = (h >> 8).double() / 16777216.0
            draws[at_b] += 1
            entry = torch.where(t0 > tmin, t0, torch.zeros_like(t0)) + tmin
            near = torch.where(hit, torch.minimum(near, entry), near)
            c, t = _brick64(case, leaves[b], descs[b], tf, org, d[at_b], t0[at_b], t1[at_b], ils, trans[at_b])
            rgb = rgb.index_add(0, at_b, c)
            trans = trans.index_copy(0, at_b, t)
            tmin = torch.where(hit, t1, tmin)
        yield px, torch.cat([rgb, 1.0 - trans[:, None]], dim=1), near


def exact(case, seed):
    kind, W, H = case["kind"], case["width"], case["height"]
    if kind not in ("train", "partials"):
        return None  # frames are RGBA8
    if case.get("views", 1) * _samples(case, W, H) > 9e8:
        return None
    descs = _descs(case)
    vol = _volume(case, seed)
    tf = torch.from_numpy(S.ramp_tf(case["tf_n"])).cuda().double()
    leaves = [V.brick_voxels(vol, q).double() for q in descs]
    if kind == "partials":
        if case["spp"] != 1 or case["crosshair"]:
            return None
        cam = _cameras(case, seed + 1, 1, W, H)[0]
        groups = [list(range(len(descs)))] if case["ranks"] == 1 else [[b] for b in range(len(descs))]
        lo = np.min([q["space_lo"] for q in descs], axis=0)
        hi = np.max([q["space_hi"] for q in descs], axis=0)
        ctr = (lo + hi) / 2
        far = float(np.linalg.norm(np.asarray(cam[0], np.float64) + ctr) + np.linalg.norm(ctr + hi))
        got = []
        with torch.no_grad():
            for grp in groups:
                img = torch.zeros((H * W, 4), dtype=torch.float64, device="cuda")
                dep = torch.ones(H * W, dtype=torch.float64, device="cuda")
                for px, rgba, near in _march64(case, [descs[b] for b in grp], [leaves[b] for b in grp], tf, cam):
                    img[px] = rgba
                    dep[px] = torch.minimum(near / far, torch.ones_like(near))
                got.append((img.reshape(H, W, 4), dep.reshape(H, W)))
        return {"images": torch.stack([g[0] for g in got]), "depth": torch.stack([g[1] for g in got]), "fb": None}
    want_tf, want_density = case["want"] != "density", case["want"] != "tf"
    tf.requires_grad_(want_tf)
    for x in leaves:
        x.requires_grad_(want_density)
    target = _targets(case, seed).double()
    imgs = torch.zeros((case["views"], H * W, 4), dtype=torch.float64, device="cuda")
    for v, cam in enumerate(_cameras(case, seed + 1, case["views"], W, H)):
        for px, rgba, _ in _march64(case, descs, leaves, tf, cam):
            imgs[v, px] = rgba.detach()
            ((rgba - target[v].reshape(-1, 4)[px]) ** 2).sum().backward()
    grads = [tf.grad] if want_tf else []
    if want_density:
        g = torch.zeros(tuple(vol.shape), dtype=torch.float64, device="cuda")
        for q, x in zip(descs, leaves):
            lo, hi = q["voxel_lo"], q["voxel_hi"]
            if x.grad is not None:
                g[lo[2]:hi[2], lo[1]:hi[1], lo[0]:hi[0]] += x.grad
        grads.append(g)
    return {"images": imgs.reshape(case["views"], H, W, 4), "grads": grads}
