"""The correction where its warps take several pieces: both grids of the sums, planar and
channels-last residuals.

Against NumPy: with a zero depth residual the two volume sums are the same (the scale
is 1 whatever their order), so every value is equal bit for bit; with one, the scale
is a float64 quotient rounded to float32, at most one rounding apart for another
order of the sums, a depth two roundings and a momentum three: within 2^-21.
"""

from __future__ import annotations

import numpy as np
import pytest
import torch

from test_gpu_coupling_pieces import _case, _dev, _same, f4

pytestmark = pytest.mark.gpu


# Pieces that fit 4 CTAs an SM, that loop there (up to 16), and that loop at 16; one long row, one tall column.
@pytest.mark.parametrize("rows,cols", [(600, 700), (1449, 1447), (2100, 2049), (1, 200_003), (300_001, 1)])
@pytest.mark.parametrize("channels_last", [False, True])
@pytest.mark.parametrize("depth_residual", [False, True])
def test_correction_on_large_grids(cuda_device, rows, cols, channels_last, depth_residual):
    from hybrid_flood_b200 import hybrid

    s, mask, _, st, rng = _case(rows, cols, rows + cols)
    st[0] = np.where(mask, st[0], f4(0))
    h, hu, hv = st
    dry = f4(s.params.dry_tolerance)
    res = (rng.normal(size=(1, 3, rows, cols)) * 0.1).astype(f4)
    if not depth_residual:
        res[:, 0] = 0.0
    dev = torch.from_numpy(res).cuda()
    if channels_last:
        dev = dev.to(memory_format=torch.channels_last)
    got = hybrid.apply_residual_correction(s, _dev(st), dev, correction_relaxation=0.25, clip_limits=[0.05] * 3)
    r = np.clip(res[0], f4(-0.05), f4(0.05))
    prov = np.where(mask, np.maximum(h + f4(0.25) * r[0], f4(0)), f4(0)).astype(f4)
    scale = f4(h[mask].sum(dtype=np.float64) / prov.sum(dtype=np.float64))
    depth = (prov * scale).astype(f4)
    wet0 = h > dry
    den = np.maximum(h, dry)
    u, v = (np.where(wet0, x / den, f4(0)).astype(f4) for x in (hu, hv))
    u, v = (u + f4(0.25) * r[1]).astype(f4), (v + f4(0.25) * r[2]).astype(f4)
    wet = mask & (depth > dry)
    want = depth, np.where(wet, depth * u, f4(0)).astype(f4), np.where(wet, depth * v, f4(0)).astype(f4)
    for g, w in zip(got, want):
        if depth_residual:
            away = np.abs(depth - dry) > 1e-6 * dry  # a depth at the dry tolerance may fall on either side
            np.testing.assert_allclose(g.cpu().numpy()[away], w[away], rtol=2.0**-21, atol=0)
        else:
            _same(g, w)
