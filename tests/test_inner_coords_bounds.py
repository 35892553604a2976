"""The limits of the unclamped coordinates (InnerCoords in
aloha_gb300/csrc/internal.h) keep every sample's voxel coordinates within a
quarter voxel of its brick: the kernels' ray, slab test and first sample
(aloha_gb300/csrc/march.cuh, steps.h) in 32-bit arithmetic, for bricks, eyes, steps
and jitters up to the limits, at the first and the last ray parameter that a march
can reach and at others between them."""
import re
import os

import numpy as np
import pytest

F = np.float32
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def limits():
    text = open(os.path.join(ROOT, "aloha_gb300", "csrc", "internal.h")).read()
    return {k: float(re.search(rf"{k} = ([0-9.]+)f", text).group(1))
            for k in ("kInnerSpace", "kInnerEye", "kInnerStep", "kInnerJitter")}


def fma(a, b, c):
    return (a.astype(np.float64) * b.astype(np.float64) + c.astype(np.float64)).astype(F)


def rays(rng, n, lim, kind):
    """Bricks (voxel range, space range), eyes and directions of unit length."""
    space, eye = lim["kInnerSpace"], lim["kInnerEye"]
    size = np.exp(rng.uniform(0, np.log(16384), (n, 3))).astype(np.int64) + (kind == "thin")
    size = np.where(rng.random((n, 3)) < (0.5 if kind == "thin" else 0.0), 1, size)
    lo = np.floor(rng.uniform(-space, space, (n, 3))).astype(np.int64)
    if kind == "corner":
        lo = np.where(rng.random((n, 3)) < 0.5, -int(space), int(space) - size)
    lo = np.clip(lo, -int(space), None)
    hi = np.minimum(lo + size, int(space))
    lo = np.minimum(lo, hi - 1)
    inset = np.where(rng.random((n, 3)) < 0.5, 0.0, rng.uniform(0, 0.4, (n, 3)))
    slo = (lo + inset * (hi - lo)).astype(F)
    shi = np.maximum((hi - inset * (hi - lo)).astype(F), np.nextafter(slo, F(np.inf)))
    slo, shi = np.maximum(slo, lo.astype(F)), np.minimum(shi, hi.astype(F))
    o = rng.uniform(-eye, eye, (n, 3))
    if kind == "corner":
        o = np.where(rng.random((n, 3)) < 0.7, eye * rng.choice([-1, 1], (n, 3)), o)
    if kind == "inside":
        o = slo + rng.random((n, 3)) * (shi - slo)
    o = o.astype(F)
    aim = slo + rng.random((n, 3)) * (shi - slo)  # towards a point of the box, or of a face or an edge of it
    aim = np.where(rng.random((n, 3)) < 0.4, np.where(rng.random((n, 3)) < 0.5, slo, shi), aim)
    d = aim - o + rng.normal(0, 1e-3, (n, 3))
    flat = rng.random((n, 3)) < 0.2
    d = np.where(flat, d * 1e-7, d)
    d = (d / np.maximum(np.linalg.norm(d, axis=1, keepdims=True), 1e-30)).astype(F)
    d = np.where(np.abs(d) < F(1e-5), F(1e-5), d)
    ok = np.isfinite(d).all(1) & (np.abs(d).max(1) > 0.5) & (slo < shi).all(1)
    return lo[ok], hi[ok], slo[ok], shi[ok], o[ok], d[ok]


@pytest.mark.parametrize("kind", ["any", "corner", "thin", "inside"])
def test_samples_stay_within_a_quarter_voxel(kind):
    lim, rng = limits(), np.random.default_rng(7)
    checked, worst = 0, 0.0
    with np.errstate(over="ignore", invalid="ignore", divide="ignore"):
        for _ in range(12):
            lo, hi, slo, shi, o, d = rays(rng, 60000, lim, kind)
            n = len(lo)
            l, h = ((slo - o) / d).astype(F), ((shi - o) / d).astype(F)
            near, far = np.minimum(l, h).max(1), np.maximum(l, h).min(1)
            tmin = np.where(rng.random(n) < 0.3, (near + rng.random(n) * (far - near)), 0.0).astype(F)
            t0, t1 = np.maximum(np.maximum(tmin, F(0)), near), np.minimum(F(1e10), far)
            dt = np.exp(rng.uniform(np.log(1e-5), np.log(lim["kInnerStep"]), n)).astype(F)
            dt = np.where(rng.random(n) < 0.3, rng.choice([0.3, 0.5, 1.0, lim["kInnerStep"]], n), dt).astype(F)
            j = lim["kInnerJitter"]
            ils = np.where(rng.random(n) < 0.5, rng.random(n), rng.choice([-j, j, -0.37 * j, 0.0], n)).astype(F)
            # first_sample_t
            k = np.floor(((t0 - dt * ils) / dt).astype(F)).astype(F)
            first = (dt * (ils + k)).astype(F)
            first = np.where(first < t0, (first + dt).astype(F), first)
            last = np.nextafter(t1, F(-np.inf))
            hit = (t0 < t1) & (first < t1)
            for t in (first, last, (first + rng.random(n).astype(F) * (last - first)).astype(F)):
                t = np.minimum(np.maximum(t, first), last)
                u = (fma(t[:, None], d, o) - lo.astype(F)).astype(F).astype(np.float64)
                out = np.maximum(-u, u - (hi - lo)).max(1)[hit]
                checked += int(hit.sum())
                worst = max(worst, float(out.max()))
    assert checked > 200000
    assert worst < 1.0 / 16.0, worst  # what internal.h states; a quarter is what the loads need
