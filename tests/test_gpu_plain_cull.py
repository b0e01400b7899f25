"""VB_CULL_NONE: the cones that find its terms change neither a bit of the sum
nor what it accepts."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from gpu_util import bl_struct, dev, geometry, get, reference_baselines, sky_struct, stage1, upstream_cosphi, zeros

pytestmark = pytest.mark.gpu


def setup(vb, nside, npix, steps, seed=3):
    (dl, dm, dn), lmn = geometry(nside)
    B = dev((vb.synthetic_sky(nside, seed=seed) / 1e5).astype(np.float32)[:npix])
    host, d = reference_baselines(30.0, 1, 42, 500, steps)
    return (sky_struct(dl, dm, dn, B, npix), bl_struct(d, host["u"].size, 28, upstream_cosphi()), lmn,
            (dl, dm, dn, B, d, host))


def plain_sum(vb, sky, bl, prec, stage):
    """The sum with every term tested at every pixel: a workspace without room for cones."""
    o = vb.Stage1Opts(precision=prec, cull=0, phase_corrected=1, blockage=1, stage_pix=stage)
    need = vb.lib().vb_stage1_workspace_bytes(C.byref(sky), C.byref(bl), C.byref(o))
    npix = sky.npix
    cones = 48 * (-(-npix // (stage or 1024)))
    ws, V = zeros(need, np.uint8), zeros(bl.n_full, np.float64)
    vb.check(vb.lib().vb_viss_halfsym(C.byref(sky), C.byref(bl), C.byref(o), ws.ptr, need - cones, V.ptr, None, None))
    return get(V, np.float64)


@pytest.mark.parametrize("nside,npix,steps,stage", [(32, 12288, 90, 0), (64, 40001, 33, 0), (64, 49152, 40, 256), (64, 49152, 40, 128)])
@pytest.mark.parametrize("prec", [1, 2, 3])
def test_cones_do_not_change_the_plain_sum(vb, gpu, nside, npix, steps, stage, prec):
    sky, bl, _, keep = setup(vb, nside, npix, steps)
    V, cnt = stage1(sky, bl, precision=prec, cull=0, stage_pix=stage)
    W = plain_sum(vb, sky, bl, prec, stage)
    assert np.array_equal(V.view(np.uint64), W.view(np.uint64))
    total = npix * (bl.n_full // 2)
    assert [int(x) for x in cnt] == [0, total, 0, total]      # every term counts as tested


def test_vectors_off_the_unit_sphere_are_tested_at_every_pixel(vb, gpu):
    """Scaled pixel vectors and endpoint norms that are not the inverse length: the cones decide nothing there."""
    sky, bl, (l, m, n), keep = setup(vb, 32, 12288, 90)
    s = np.ones(12288, np.float32)
    s[5000:9000] = 1.3
    arrs = [dev(a * s) for a in (l, m, n)]
    sky.l, sky.m, sky.n = (a.ptr for a in arrs)
    inv = dev(get(keep[4]["invn1"]) * np.where(np.arange(bl.n_full) % 3 == 0, np.float32(0.4), np.float32(1)).astype(np.float32))
    bl.invn1 = inv.ptr
    V, _ = stage1(sky, bl, precision=vb.PREC_FP32_FP64PH, cull=0)
    W = plain_sum(vb, sky, bl, vb.PREC_FP32_FP64PH, 0)
    assert np.array_equal(V.view(np.uint64), W.view(np.uint64))
