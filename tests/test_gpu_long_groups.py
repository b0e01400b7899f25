"""Stage 2 with member sampling (k_recon_members) on groups of about one, two and more than
two buffers of members (256 each): the part-by-part walk of occ_mode 0 against the FP64 oracle.

Tolerance: as in test_gpu_stage2.py (FP64: float32 output; FP32 sum: 1e-5).
"""
from __future__ import annotations

import numpy as np
import pytest

from conftest import rel_err
from gpu_util import bl_struct, dev, geometry, reference_baselines, sky_struct, stage2, upstream_cosphi

pytestmark = pytest.mark.gpu

SIZES = [1, 255, 256, 257, 2, 511, 512, 513, 3]   # members of each cell; the rest share one


@pytest.mark.parametrize("mirror", [1, 0])
@pytest.mark.parametrize("occ", [0, 1, 3])
@pytest.mark.parametrize("prec,tol", [("fp64", 2e-7), ("fp32_fp64phase", 1e-5)])
def test_groups_longer_than_the_buffer(vb, gpu, orc, mirror, occ, prec, tol):
    nside, steps = 16, 128
    npix = 12 * nside * nside
    (dl, dm, dn), (l, m, n) = geometry(nside)
    B = np.ones(npix, np.float32)
    dB = dev(B)
    host, d = reference_baselines(300.0, 1, 42, 100, steps)
    nh = host["u"].size // 2
    cell = np.full(nh, len(SIZES))
    order = np.random.default_rng(4).permutation(nh)       # members of a cell scattered over steps and pairs
    for k, at in enumerate(np.cumsum([0] + SIZES[:-1])):
        cell[order[at:at + SIZES[k]]] = k
    f = (np.arange(nh) // 28) * 56 + np.arange(nh) % 28
    bl_max, lam = 1000.0, 10.0                             # cells of 6.25 wavelengths
    for key, x in (("u", 6.25 * (cell + 1)), ("v", 6.25 * (cell % 4))):
        host[key][f] = x
        host[key][f + 28] = -x
        d[key] = dev(host[key])
    sky = sky_struct(dl, dm, dn, dB, npix)
    bl = bl_struct(d, host["u"].size, 28, upstream_cosphi())
    V = np.random.default_rng(5).normal(size=(nh, 2)).astype(np.float32)
    kw = dict(mirror=mirror, blockage=1, occ_mode=occ, lam=lam, bl_max=bl_max, grid_res=33)
    pm = {"fp64": vb.PREC_FP64, "fp32_fp64phase": vb.PREC_FP32_FP64PH}[prec]
    Cd, W, params, _ = stage2(sky, bl, dev(V), [0], [steps], precision=pm, **kw)
    Co, Wo, sp = orc.stage2(dict(B=B, l=l, m=m, n=n), dict(host, cosphi=upstream_cosphi()), V, [0], [steps], precision=1, **kw)
    assert params[0]["nuniq"] == sp["nuniq"][0] == (len(SIZES) + 1) * (1 if mirror else 2)
    assert np.array_equal(W, Wo)
    emax, erms = rel_err(Cd, Co)
    assert emax <= tol and erms <= tol, (emax, erms)
