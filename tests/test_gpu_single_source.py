"""Factored sums with one term that matters: a sky of one source (stage 1), one visibility
(stage 2).  Errors then cannot cancel, so this is the largest error of a term.

The pairs move along tracks of one direction at many speeds, so that every polynomial is
met at the ends of its range.  Stage 1: the source is the pixel that lies farthest along the
tracks (across them where they are noisy) from its block's centre; stage 2: the
visibility is the last of a cluster.

Tolerance for |exp(i phi)|: half a step of the 2^-23-turn phase grid 3.7e-7, the angle in
float32 2.4e-7 and its fl(2 pi) 1.7e-7, the SFU's sine and cosine 6e-7, polynomials
6e-7 and their float sums 5e-7 (powers up to 2.5^n / n!; 8e-7 and 1e-7 where residuals
lead), 2.5e-6 in all; the per-term kernel's own bound, with three roundings of the
phase, is 2.1e-6.  Stage 2:
polynomials 1.5e-7 and their float sums 2e-7, 1.8e-6 in all.
"""
from __future__ import annotations

import numpy as np
import pytest

from gpu_util import dev, geometry, sky_struct, stage1, stage2, zeros

pytestmark = pytest.mark.gpu

TOL = 2.5e-6


def tracks(vb, steps, speeds, axis, across, bend, noise=0.0):
    """Signed baselines of len(speeds) pairs: straight tracks with a bend of `bend` radians over 128 steps, off
    them by up to `noise` wavelengths (the first pair by little, the last by that)."""
    n = len(speeds)
    k = np.arange(steps)[:, None] - 0.5 * steps
    s = np.asarray(speeds)[None, :] * k
    c = s * (bend / 128) * k * 0.5
    start = np.stack([np.linspace(-300, 250, n), np.linspace(200, 330, n), np.linspace(30, -90, n)], 1)
    u = start[None] + s[:, :, None] * axis + c[:, :, None] * across
    u = u + np.random.default_rng(8).uniform(-1, 1, u.shape) * (noise * np.linspace(0.02, 1, n))[None, :, None]
    full = np.concatenate([-u, u], 1).reshape(-1, 3).astype(np.float32)
    bl = vb.Baselines(n_full=full.shape[0], nbl=n)
    d = {key: dev(np.ascontiguousarray(full[:, i])) for i, key in enumerate("uvw")}
    for key, b in d.items():
        setattr(bl, key, b.ptr)
    return bl, d


@pytest.mark.parametrize("nside,bend,noise,fastest", [(512, 0.0, 0, 3.0), (512, 0.05, 0, 3.0), (512, 0.2, 0, 3.0), (256, 0.4, 0, 3.0),
                                                      (128, 0.05, 0, 3.0), (512, 0.02, 0.008, 0.04), (512, 0.02, 0.005, 0.4)])
def test_one_source(vb, gpu, nside, bend, noise, fastest):
    npix = min(12 * nside * nside, 1 << 20)
    (dl, dm, dn), lmn = geometry(nside)
    s = np.stack([a[:npix] for a in lmn], 1).astype(np.float64)
    worst = 0.0
    for block in (64, 256, 1024):
        t = (s.reshape(-1, block, 3) - s.reshape(-1, block, 3).mean(1, keepdims=True)).reshape(-1, 3)
        for p in np.argsort(-(t * t).sum(1))[:6:3]:
            axis = t[p] / np.linalg.norm(t[p])
            across = np.cross(s[p], axis)
            if noise:                     # the source lies across the tracks: the residuals count
                axis, across = across, axis
            steps = 128 * -(-(6_100_000_000 // (npix * 56)) // 128)
            bl, keep = tracks(vb, max(steps, 256), np.geomspace(0.02, fastest, 56), axis, across, bend, noise)
            B = np.zeros(npix, np.float32)
            B[p] = 1.0
            dB = dev(B)
            sky = sky_struct(dl, dm, dn, dB, npix)
            V, _ = stage1(sky, bl, precision=vb.PREC_FP32_FP64PH, cull=0, blockage=0)
            V64, _ = stage1(sky, bl, precision=vb.PREC_FP64, cull=0, blockage=0)
            e = (V - V64).reshape(-1, 2)
            worst = max(worst, float(np.hypot(e[:, 0], e[:, 1]).max()))
    print("largest error of a term", worst)
    assert worst <= TOL


def test_one_visibility(vb, gpu):
    npix, steps, pairs = 2200000, 500, 28
    (dl, dm, dn), _ = geometry(512)
    sky = sky_struct(dl, dm, dn, dl, npix)
    axis, across = np.array([0.8, 0.6, 0.0]), np.array([-0.6, 0.8, 0.0])
    # cells of 0.1 wavelengths: each step of a track has its own, clusters of 32 steps
    bl, keep = tracks(vb, steps, np.geomspace(0.15, 0.7, pairs), axis, across, 0.02)
    ends = [zeros(bl.n_full) for _ in range(8)]
    for k, b in zip(("x1", "y1", "z1", "invn1", "x2", "y2", "z2", "invn2"), ends):
        setattr(bl, k, b.ptr)
    kw = dict(mirror=1, blockage=0, lam=1.0, bl_max=819.2, grid_res=16385)
    worst, seen = 0.0, 0
    for pair in range(pairs):
        V = np.zeros((steps * pairs, 2), np.float32)
        V[(160 + 31 * (pair % 2)) * pairs + pair] = (0.8, -0.6)
        dV = dev(V)
        C1, _, p1, _ = stage2(sky, bl, dV, [0], [steps], precision=vb.PREC_FP32_FP64PH, **kw)
        C64, _, p64, _ = stage2(sky, bl, dV, [0], [steps], precision=vb.PREC_FP64, **kw)
        assert p1 == p64
        if not C64.any():
            continue          # (off the grid)
        seen += 1
        worst = max(worst, float(np.abs(C1.astype(np.float64) - C64).max()) * p64[0]["nuniq"])
    print("largest error of a term", worst)
    assert seen > pairs // 2 and worst <= 1.8e-6
