"""A small call's work items take parts of a cull tile: the same terms and the
same sum as with whole tiles."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from gpu_util import bl_struct, dev, geometry, get, reference_baselines, sky_struct, stage1, tile_meta, upstream_cosphi, zeros

pytestmark = pytest.mark.gpu

# |sum of the terms' brightness| times this bounds the difference: FP64 sums of up to
# 2^16 terms reordered; FP32 partial sums of up to 1024 terms (both sides round)
TOL = {0: 2.0 ** 16 * 2.0 ** -53 * 2, 1: 1024 * 2.0 ** -24 * 2, 2: 1024 * 2.0 ** -24 * 2}


@pytest.mark.parametrize("nside,npix,steps,cull,tile,refine", [
    (32, 12288, 7, 1, 256, 0),         # 128-pixel parts, one warp of the tile idle
    (64, 40001, 33, 1, 4096, 0),       # 256-pixel sub-tiles, a last part of 65 pixels
    (64, 49152, 19, 1, 16384, 0),
    (64, 49152, 19, 1, 16384, 1024),   # sub-tiles wider than a part
    (64, 40001, 33, 2, 0, 0),
    (64, 32769, 20, 0, 0, 0),          # one pixel in the last part
])
def test_parts_of_a_tile(vb, gpu, nside, npix, steps, cull, tile, refine):
    (dl, dm, dn), _ = geometry(nside)
    host_B = (vb.synthetic_sky(nside, seed=5) / 1e5).astype(np.float32)[:npix]
    B = dev(host_B)
    host, d = reference_baselines(30.0, 1, 42, 500, steps)
    meta = (tile, tile_meta(tile, dl, dm, dn, npix)) if cull == 1 else None
    sky, bl = sky_struct(dl, dm, dn, B, npix, meta), bl_struct(d, host["u"].size, 28, upstream_cosphi())
    kw = dict(cull=cull, refine_pix=refine)
    whole = {1: tile, 2: 1024, 0: 1024}[cull]
    for prec, tol in ((vb.PREC_FP64, TOL[0]), (vb.PREC_FP32_FP64PH, TOL[1]), (vb.PREC_FP32_DSPH, TOL[2])):
        V, cnt = stage1(sky, bl, precision=prec, **kw)
        W, ref = stage1(sky, bl, precision=prec, chunk_pix=whole, **kw)
        assert np.max(np.abs(V - W)) <= tol * host_B.sum(dtype=np.float64)
        assert [int(x) for x in cnt] == [int(x) for x in ref]


def test_parts_need_no_more_room_than_whole_tiles(vb, gpu):
    """A workspace that holds whole tiles is still enough."""
    (dl, dm, dn), _ = geometry(64)
    B = dev((vb.synthetic_sky(64, seed=5) / 1e5).astype(np.float32))
    host, d = reference_baselines(30.0, 1, 42, 500, 19)
    meta = (16384, tile_meta(16384, dl, dm, dn, 49152))
    sky, bl = sky_struct(dl, dm, dn, B, 49152, meta), bl_struct(d, host["u"].size, 28, upstream_cosphi())
    o = vb.Stage1Opts(precision=vb.PREC_FP64, cull=1, phase_corrected=1, blockage=1)
    need = vb.lib().vb_stage1_workspace_bytes(C.byref(sky), C.byref(bl), C.byref(o))
    o.chunk_pix = 16384
    small = vb.lib().vb_stage1_workspace_bytes(C.byref(sky), C.byref(bl), C.byref(o))
    assert small < need
    out = []
    for chunk, size in ((16384, need), (0, small)):
        o.chunk_pix = chunk
        ws, V = zeros(need, np.uint8), zeros(bl.n_full, np.float64)
        vb.check(vb.lib().vb_viss_halfsym(C.byref(sky), C.byref(bl), C.byref(o), ws.ptr, size, V.ptr, None, None))
        out.append(get(V, np.float64))
    assert np.array_equal(out[0], out[1])
