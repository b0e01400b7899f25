"""Stage 2 with clusters of uv groups (vb_track2.cu) on segment tables whose ranges
overlap, repeat a start, are out of order or leave the day: what the FP64 build gives, which sums
every group by itself, the same bits on every call, and each group once (W).

Tolerance: as in test_gpu_clusters.py (4e-7 rms a term, 1.5e-6 for the largest).
"""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from conftest import rel_err
from gpu_util import dev, get, stage2, zeros
from test_gpu_clusters import TOL, setup

pytestmark = pytest.mark.gpu


def per_group(vb, sky, bl, dV, t0, tl, lam):
    """The image with a workspace that has no room for clusters."""
    o = vb.Stage2Opts(mirror=1, blockage=1, occ_mode=2, precision=vb.PREC_FP32_FP64PH, cull=2, grid_res=0, bl_max=100e3, lambda_=lam)
    need = vb.lib().vb_stage2_workspace_bytes(bl.n_full // 2, len(t0), sky.npix, C.byref(o))
    ws, Cb, Wb = zeros(need, np.uint8), zeros(sky.npix), zeros(sky.npix, np.uint32)
    a, b = dev(np.asarray(t0, np.int32)), dev(np.asarray(tl, np.int32))
    vb.check(vb.lib().vb_recon_batched(C.byref(sky), C.byref(bl), dV.ptr, len(t0), a.ptr, b.ptr, C.byref(o), ws.ptr,
                                       need - 32 * (sky.npix // 64), Cb.ptr, Wb.ptr, None, None, None))
    return get(Cb)


@pytest.mark.parametrize("t0,tl,clusters", [
    ([0, 250], [250, 250], True),
    ([0, 200], [250, 300], True),
    ([0, 100, 200], [300, 300, 300], True),
    ([0, 0, 150], [300, 500, 350], True),        # the first entry has no step of its own
    ([250, 0], [250, 250], True),                # out of order
    ([100, 100, 350], [120, 60, 150], True),     # steps before the first entry and between two
    ([0, 300], [300, 400], True),                # past the day's end
    ([-50, 250], [300, 250], True),              # from before its start
])
def test_clusters_on_any_segment_table(vb, gpu, t0, tl, clusters):
    sky, bl, V, keep = setup(vb, 512, 2200001, 300.0, 500, 1)
    dV = dev(V)
    kw = dict(mirror=1, blockage=1, cull=2, lam=300.0)
    C1, W1, p1, c1 = stage2(sky, bl, dV, t0, tl, precision=vb.PREC_FP32_FP64PH, **kw)
    for _ in range(3):
        C2, W2, _, _ = stage2(sky, bl, dV, t0, tl, precision=vb.PREC_FP32_FP64PH, **kw)
        assert np.array_equal(C1.view(np.uint32), C2.view(np.uint32)) and np.array_equal(W1, W2)
    # the clusters were in use: other bits than without
    assert clusters != np.array_equal(C1.view(np.uint32), per_group(vb, sky, bl, dV, t0, tl, 300.0).view(np.uint32))
    C64, W64, p64, c64 = stage2(sky, bl, dV, t0, tl, precision=vb.PREC_FP64, ppt=4, **kw)
    assert np.array_equal(W1, W64) and p1 == p64 and np.array_equal(c1, c64)
    assert max(rel_err(C1, C64)) <= TOL, rel_err(C1, C64)
