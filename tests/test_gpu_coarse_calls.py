"""Skies of up to four 1024-pixel tiles take fewer parts and no cones up to a line (4095 and
4096 pixels lie on its two sides): the terms and the sum of whole tiles and of the exact
tile classes, whichever way a call is cut.

Tolerance: |sum of the terms' brightness| times the roundings of FP32 partial sums of up to
1024 terms on both sides (FP64: sums of up to 2^16 terms reordered)."""
from __future__ import annotations

import numpy as np
import pytest

from gpu_util import bl_struct, dev, geometry, reference_baselines, sky_struct, stage1, upstream_cosphi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("npix,steps", [(1500, 200), (3072, 240), (3072, 1800), (4095, 300), (4096, 300), (4095, 3300)])
def test_coarse_skies(vb, gpu, npix, steps):
    nside = 32 if npix > 3072 else 16
    (dl, dm, dn), _ = geometry(nside)
    host_B = (vb.synthetic_sky(nside, seed=5) / 1e5).astype(np.float32)[:npix]
    host, d = reference_baselines(30.0, 1, 42, 500, steps)
    keep = dev(host_B)
    sky, bl = sky_struct(dl, dm, dn, keep, npix), bl_struct(d, host["u"].size, 28, upstream_cosphi())
    total = npix * (bl.n_full // 2)
    for prec, tol in ((vb.PREC_FP64, 2.0 ** 16 * 2.0 ** -53 * 2), (vb.PREC_FP32_FP64PH, 1024 * 2.0 ** -24 * 2)):
        V = {}
        for cull in (0, 2):
            for chunk in (0, 1024):
                V[cull, chunk], cnt = stage1(sky, bl, precision=prec, cull=cull, chunk_pix=chunk)
                assert int(cnt[3]) == total and int(cnt[0] + cnt[1] + cnt[2]) == total
        for k in V:
            assert np.max(np.abs(V[k] - V[0, 0])) <= tol * host_B.sum(dtype=np.float64), k
