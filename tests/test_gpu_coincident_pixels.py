"""Skies whose pixel blocks hold one direction many times over: the factored sums
(vb_track.cu, vb_track2.cu) divide by the blocks' radius, which is then zero.

Tolerance: pixels of one direction share one rounding of the phase (1.5 steps of its
2^-23-turn grid, 1.1e-6 rad) and one of the SFU (angle 4e-7, sine and cosine 6e-7),
so that the largest error is that of a term, under 3e-6, and the 2-norm's its rms
(4.4e-7 measured), under 1e-6.
"""
from __future__ import annotations

import numpy as np
import pytest

from conftest import rel_err
from gpu_util import bl_struct, dev, geometry, reference_baselines, sky_struct, stage1, stage2, tile_meta, upstream_cosphi

pytestmark = pytest.mark.gpu


def sky_of_copies(nside, npix, copies):
    """npix pixels, `copies` in a row of each of the sky's first directions."""
    _, lmn = geometry(nside)
    a = [dev(np.repeat(x[:-(-npix // copies)], copies)[:npix]) for x in lmn]
    assert a[0].nbytes == 4 * npix
    return a


@pytest.mark.parametrize("nside,copies,cull,blockage", [(64, 64, 1, 1), (64, 64, 0, 1), (16, 1024, 0, 0), (16, 1 << 18, 2, 1)])
def test_stage1_of_coincident_pixels(vb, gpu, nside, copies, cull, blockage):
    npix = 196608
    dl, dm, dn = sky_of_copies(nside, npix, copies)
    host, d = reference_baselines(300.0, 1, 42, 100, 1100)
    dB = dev(np.random.default_rng(1).uniform(0, 1, npix).astype(np.float32))
    tiles = tile_meta(256, dl, dm, dn, npix)
    sky = sky_struct(dl, dm, dn, dB, npix, (256, tiles))
    bl = bl_struct(d, host["u"].size, host["nbl"], upstream_cosphi())
    V, _ = stage1(sky, bl, precision=vb.PREC_FP32_FP64PH, cull=cull, blockage=blockage)
    V64, _ = stage1(sky, bl, precision=vb.PREC_FP64, cull=cull, blockage=blockage)
    emax, erms = rel_err(V, V64)
    assert emax <= 3e-6 and erms <= 1e-6, (emax, erms)


@pytest.mark.parametrize("nside,copies", [(32, 256), (1, 1 << 18)])
def test_stage2_of_coincident_pixels(vb, gpu, nside, copies):
    npix = 2200000
    dl, dm, dn = sky_of_copies(nside, npix, copies)
    host, d = reference_baselines(300.0, 1, 42, 100, 500)
    sky = sky_struct(dl, dm, dn, dl, npix)
    bl = bl_struct(d, host["u"].size, host["nbl"], upstream_cosphi())
    dV = dev(np.random.default_rng(2).normal(size=host["u"].size).astype(np.float32))
    kw = dict(mirror=1, blockage=1, cull=2, lam=300.0)
    C1, W1, _, _ = stage2(sky, bl, dV, [0], [500], precision=vb.PREC_FP32_FP64PH, **kw)
    C64, W64, _, _ = stage2(sky, bl, dV, [0], [500], precision=vb.PREC_FP64, **kw)
    assert np.array_equal(W1, W64)
    emax, erms = rel_err(C1, C64)
    assert emax <= 3e-6 and erms <= 1e-6, (emax, erms)
