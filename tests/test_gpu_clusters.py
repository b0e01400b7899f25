"""Stage 2 over clusters of uv groups (vb_track2.cu): the image, W and the term
counters against the FP64 reconstruction, which sums every group by itself.

Tolerance: a term carries at most about 4e-7 rms (2^-23-turn phase grid, SFU
sine and cosine, polynomial below 1e-7), and so does a sum of independent terms
in the 2-norm; 1.5e-6 leaves room for the largest value.
"""
from __future__ import annotations

import numpy as np
import pytest

from conftest import rel_err
from gpu_util import bl_struct, dev, geometry, reference_baselines, sky_struct, stage2, synthetic_baselines, upstream_cosphi

pytestmark = pytest.mark.gpu

TOL = 1.5e-6


def setup(vb, nside, npix, lam, steps, day, earth=0):
    (dl, dm, dn), _ = geometry(nside)
    B = dev(np.ones(npix, np.float32))
    if earth:
        host, d = synthetic_baselines(earth, steps, lam)
    else:
        host, d = reference_baselines(lam, day, 42, 100, steps)
    sky = sky_struct(dl, dm, dn, B, npix)
    bl = bl_struct(d, host["u"].size, host["nbl"], upstream_cosphi(), bool(earth))
    rng = np.random.default_rng(3)
    nh = host["u"].size // 2
    nbl = host["nbl"]
    f = (np.arange(nh) // nbl) * 2 * nbl + np.arange(nh) % nbl
    ph = 2 * np.pi * (0.3 * host["u"][f].astype(np.float64) - 0.5 * host["v"][f] + 0.81 * host["w"][f])
    V = np.stack([np.cos(ph), -np.sin(ph)], 1) + 0.2 * rng.normal(size=(nh, 2))
    return sky, bl, V.astype(np.float32), (dl, dm, dn, B, d)


@pytest.mark.parametrize("nside,npix,lam,steps,day,earth,segs,mirror,blockage,cull", [
    (512, 3000001, 300.0, 500, 1, 0, 2, 1, 1, 2),     # ragged sky, uneven segments
    (512, 1200000, 30.0, 1000, 3, 0, 1, 1, 1, 2),     # long tracks: full clusters
    (512, 800000, 300.0, 700, 8, 0, 3, 0, 1, 0),     # signed set, halves of clusters, no block culling
    (512, 1800000, 300.0, 300, 5, 0, 1, 0, 0, 0),     # group averages
    (512, 2200000, 300.0, 400, 1, 9, 2, 1, 1, 2),     # Earth orbits: few clusters or none
])
def test_clusters_vs_fp64_reconstruction(vb, gpu, nside, npix, lam, steps, day, earth, segs, mirror, blockage, cull):
    sky, bl, V, keep = setup(vb, nside, npix, lam, steps, day, earth)
    cuts = np.linspace(0, steps, segs + 1).astype(np.int32)
    dV = dev(V)
    kw = dict(mirror=mirror, blockage=blockage, cull=cull, lam=lam, ppt=2, grid_res=513 if earth else 0)
    C1, W1, p1, c1 = stage2(sky, bl, dV, cuts[:-1], np.diff(cuts), precision=vb.PREC_FP32_FP64PH, **kw)
    C2, W2, p2, c2 = stage2(sky, bl, dV, cuts[:-1], np.diff(cuts), precision=vb.PREC_FP32_FP64PH, **kw)
    assert np.array_equal(C1.view(np.uint32), C2.view(np.uint32)) and np.array_equal(W1, W2)
    C64, W64, p64, c64 = stage2(sky, bl, dV, cuts[:-1], np.diff(cuts), precision=vb.PREC_FP64, **kw)
    assert max(rel_err(C1, C64)) <= TOL, rel_err(C1, C64)
    assert np.array_equal(W1, W64) and np.array_equal(c1, c64) and p1 == p64


def test_one_infinite_visibility_stays_in_its_own_pixels(vb, gpu):
    """An infinite V makes exactly the pixels that see its group non-finite."""
    sky, bl, V, keep = setup(vb, 512, 1200000, 30.0, 1000, 3)
    V[5000] = np.inf
    dV = dev(V)
    kw = dict(mirror=1, blockage=1, cull=2, lam=30.0)
    C1, W1, _, _ = stage2(sky, bl, dV, [0], [1000], precision=vb.PREC_FP32_FP64PH, **kw)
    C64, W64, _, _ = stage2(sky, bl, dV, [0], [1000], precision=vb.PREC_FP64, **kw)
    assert np.array_equal(W1, W64) and np.array_equal(np.isfinite(C1), np.isfinite(C64))


def test_overlapping_segment_table(vb, gpu):
    """A segment table whose ranges overlap or run past the day gives what the FP64 build gives."""
    sky, bl, V, keep = setup(vb, 512, 2000003, 300.0, 500, 1)
    dV = dev(V)
    kw = dict(mirror=1, blockage=1, cull=2, lam=300.0)
    for t0, tl in (([0, 200], [250, 300]),):
        C1, W1, p1, _ = stage2(sky, bl, dV, t0, tl, precision=vb.PREC_FP32_FP64PH, **kw)
        C64, W64, p64, _ = stage2(sky, bl, dV, t0, tl, precision=vb.PREC_FP64, **kw)
        assert np.array_equal(W1, W64) and p1 == p64 and max(rel_err(C1, C64)) <= TOL
