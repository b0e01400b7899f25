"""Stage 1 over track groups (vb_track.cu): the factored sum against the plain
FP64 sum, and its inclusion decisions against the per-pixel masks.

Tolerance: a term carries at most about 4e-7 rms (2^-23-turn phase grid, SFU
sine and cosine, truncation below 1e-7), so that a sum of independent terms is
off by about that much in the 2-norm; 1.5e-6 leaves room for the largest value.
"""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from conftest import rel_err
from gpu_util import (bl_struct, dev, geometry, get, reference_baselines, sky_struct, stage1, synthetic_baselines,
                      tile_classes, tile_meta, upstream_cosphi, zeros)

pytestmark = pytest.mark.gpu

TOL = 1.5e-6
CULL = {"none": 0, "tilecone": 1, "exact": 2}


def setup(vb, nside, npix, lam, steps, day=5, earth=0, tile=256, B=None):
    """Sky of NEST pixels [0, npix) and the baselines of `steps` steps, on the device."""
    full = 12 * nside * nside
    (dl, dm, dn), (l, m, n) = geometry(nside)
    if B is None:
        B = (vb.synthetic_sky(nside, seed=3).astype(np.float64) * (4 * np.pi / full)).astype(np.float32)
    dB = dev(B[:npix])
    if earth:
        host, d = synthetic_baselines(earth, steps, lam)
        cp, per_end = upstream_cosphi(), True
    else:
        host, d = reference_baselines(lam, day, 42, 100, steps)
        cp, per_end = upstream_cosphi(), False
    tiles = tile_meta(tile, dl, dm, dn, npix)
    sky = sky_struct(dl, dm, dn, dB, npix, (tile, tiles))
    bl = bl_struct(d, host["u"].size, host["nbl"], cp, per_end)
    return dict(sky=sky, bl=bl, host=host, d=d, l=l[:npix], m=m[:npix], n=n[:npix], cosphi=cp, per_end=per_end,
                keep=(dl, dm, dn, dB, tiles))


@pytest.mark.parametrize("nside,npix,steps,lam,day,earth,tile,cull,blockage,corrected", [
    (128, 196608, 1100, 300.0, 1, 0, 256, "tilecone", 1, 1),      # whole sky, steps not a multiple of a group
    (128, 196608, 1152, 300.0, 1, 0, 64, "tilecone", 1, 1),       # the smallest cull tiles: 64-pixel blocks only
    (512, 3145728, 97, 300.0, 3, 0, 4096, "tilecone", 1, 0),      # one short group a pair, raw phase
    (256, 600007, 385, 30.0, 2, 0, 1024, "exact", 1, 1),         # ragged sky, a group of one step
    (256, 600007, 385, 30.0, 2, 0, 1024, "none", 1, 0),
    (128, 196608, 1100, 300.0, 8, 0, 256, "none", 0, 1),          # no occlusion
    (256, 786432, 386, 300.0, 1, 7, 1024, "tilecone", 1, 1),     # Earth orbits: some groups factored, some left
    (64, 49152, 4500, 300.0, 1, 0, 1024, "tilecone", 1, 1),      # coarse sky
])
def test_track_groups_vs_fp64_sum(vb, gpu, nside, npix, steps, lam, day, earth, tile, cull, blockage, corrected):
    c = setup(vb, nside, npix, lam, steps, day, earth, tile)
    kw = dict(cull=CULL[cull], blockage=blockage, phase_corrected=corrected)
    V, cnt, flags = stage1(c["sky"], c["bl"], precision=vb.PREC_FP32_FP64PH, want_flags=True, **kw)
    V2, cnt2 = stage1(c["sky"], c["bl"], precision=vb.PREC_FP32_FP64PH, **kw)
    assert np.array_equal(V.view(np.uint64), V2.view(np.uint64)) and np.array_equal(cnt, cnt2)
    assert flags == 0
    V64, _ = stage1(c["sky"], c["bl"], precision=vb.PREC_FP64, **kw)
    emax, erms = rel_err(V, V64)
    assert emax <= TOL and erms <= TOL, (emax, erms)
    assert int(cnt[3]) == npix * (c["bl"].n_full // 2) and int(cnt[0] + cnt[1] + cnt[2]) == int(cnt[3])


@pytest.mark.parametrize("cull", ["none", "tilecone", "exact"])
def test_track_groups_include_the_masked_terms(vb, gpu, orc, cull):
    """u = v = w = 0 and B = 1: V is the number of included pixels of each baseline."""
    nside, steps, tile = 128, 1100, 256
    c = setup(vb, nside, 196608, 300.0, steps, B=np.ones(196608, np.float32))
    nh = c["bl"].n_full // 2
    zero = zeros(c["bl"].n_full)
    c["bl"].u = c["bl"].v = c["bl"].w = zero.ptr
    V, _ = stage1(c["sky"], c["bl"], precision=vb.PREC_FP32_FP64PH, cull=CULL[cull])
    ih = np.arange(0, nh, 97)
    f = (ih // 28) * 56 + ih % 28
    h = c["host"]
    inc = np.ones((ih.size, 196608), np.uint8)
    for e in "12":
        inc &= orc.occlusion_mask(c["l"], c["m"], c["n"], *(np.ascontiguousarray(h[k + e][f]) for k in ("x", "y", "z", "invn")),
                                  c["cosphi"])
    if cull == "tilecone":
        cls, _ = tile_classes(c["sky"], c["bl"], cull=CULL[cull])
        per = np.repeat(cls[ih], tile, axis=1)
        inc = np.where(per == 1, 1, np.where(per == 0, 0, inc))
    want = inc.sum(1)
    got = V[0::2][ih]
    assert np.abs(got - want).max() < 0.4, int(np.abs(np.rint(got) - want).max())


def test_track_groups_leave_irregular_input_to_the_per_term_kernel(vb, gpu):
    """An infinite pixel, shuffled pixels and scattered baselines: what the plain sum gives."""
    c = setup(vb, 128, 196608, 300.0, 1100)
    B = get(c["keep"][3])
    B[1234] = np.inf
    dB = dev(B)
    c["sky"].B = dB.ptr
    V, _ = stage1(c["sky"], c["bl"], precision=vb.PREC_FP32_FP64PH, cull=0)
    V64, _ = stage1(c["sky"], c["bl"], precision=vb.PREC_FP64, cull=0)
    assert np.array_equal(np.isfinite(V), np.isfinite(V64))
    B[1234] = 0.0
    perm = np.random.default_rng(1).permutation(196608)
    arrs = [dev(a[perm]) for a in (B, c["l"], c["m"], c["n"])]
    c["sky"].B, c["sky"].l, c["sky"].m, c["sky"].n = (a.ptr for a in arrs)
    V, _ = stage1(c["sky"], c["bl"], precision=vb.PREC_FP32_FP64PH, cull=0)
    V64, _ = stage1(c["sky"], c["bl"], precision=vb.PREC_FP64, cull=0)
    assert max(rel_err(V, V64)) <= TOL
    c = setup(vb, 128, 196608, 300.0, 1100)
    rng = np.random.default_rng(2)
    uvw = [dev(rng.uniform(-300, 300, c["bl"].n_full).astype(np.float32)) for _ in range(3)]
    c["bl"].u, c["bl"].v, c["bl"].w = (a.ptr for a in uvw)
    V, _ = stage1(c["sky"], c["bl"], precision=vb.PREC_FP32_FP64PH, cull=1)
    V64, _ = stage1(c["sky"], c["bl"], precision=vb.PREC_FP64, cull=1)
    assert max(rel_err(V, V64)) <= TOL


def test_workspace_of_the_per_term_kernel_still_serves(vb, gpu):
    """A workspace that only the per-term kernel fits in is accepted, as is the fixed-scratch entry."""
    c = setup(vb, 128, 196608, 300.0, 1100)
    o = vb.Stage1Opts(precision=vb.PREC_FP32_FP64PH, cull=1, phase_corrected=1, blockage=1)
    sky, bl = c["sky"], c["bl"]
    need = vb.lib().vb_stage1_workspace_bytes(C.byref(sky), C.byref(bl), C.byref(o))
    nh = bl.n_full // 2
    nodes = sum(32 * -(-196608 // p) for p in (64, 256, 1024))
    ws, V, Vn = zeros(need, np.uint8), zeros(2 * nh, np.float64), zeros(2 * nh, np.float64)
    vb.check(vb.lib().vb_viss_halfsym(C.byref(sky), C.byref(bl), C.byref(o), ws.ptr, need - nodes, V.ptr, None, None))
    vb.check(vb.lib().vb_viss_halfsym_noalloc(C.byref(sky), C.byref(bl), C.byref(o), Vn.ptr, None, None, None))
    V64, _ = stage1(sky, bl, precision=vb.PREC_FP64, cull=1)
    assert max(rel_err(get(V, np.float64), V64)) <= TOL and max(rel_err(get(Vn, np.float64), V64)) <= TOL
