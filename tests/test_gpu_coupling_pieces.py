"""Features, correction and output fields at the edges of a warp's 128-column piece.

Against the same formulas in NumPy float32, operation by operation: equal bits
(the feature bfloat16s are the rounded float32s).  The values include what a
branch-free division could get wrong: zeros of both signs, subnormals, values
near the ends of the float range, infinities and NaN.  The correction's volume
scale is a float64 sum rounded to float32, whose order may differ: with a zero
residual and non-negative depths the two sums are the same and the scale is 1.
"""

from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

f4 = np.float32


def _case(rows, cols, seed):
    rng = np.random.default_rng(seed)
    mask = rng.random((rows, cols)) < 0.9
    mask.flat[0] = True
    kw = dict(resolution_m=2.0, rainfall_times_s=np.asarray([0, 600], f4), rainfall_rates_m_s=np.asarray([1e-5, 1e-5], f4),
              boundary=(0, 0, 0, 0))
    from hybrid_flood_b200.solver import B200ShallowWaterSolver

    bed = rng.uniform(0, 3, (rows, cols)).astype(f4)
    s = B200ShallowWaterSolver(bed, np.full((rows, cols), 0.03, f4), mask, **kw)
    h = (rng.uniform(0, 1, (rows, cols)) * (rng.random((rows, cols)) < 0.7)).astype(f4)
    hu, hv = ((rng.normal(0, 1, (2, rows, cols)) * (rng.random((2, rows, cols)) < 0.8))).astype(f4)
    return s, mask, bed, [h, hu, hv], rng


def _dev(st, pad=0):
    from hybrid_flood_b200.solver import SWEState

    out = []
    for a in st:
        w = torch.full((a.shape[0], a.shape[1] + pad), 9.0, device="cuda")
        w[:, : a.shape[1]] = torch.from_numpy(a)
        out.append(w[:, : a.shape[1]])
    return SWEState(*out)


def _same(got, want):
    got = np.asarray(got.cpu() if isinstance(got, torch.Tensor) else got)
    assert got.shape == want.shape
    ok = (got.view(np.uint32) == want.astype(f4).view(np.uint32)) | (np.isnan(got) & np.isnan(want))
    assert ok.all(), (np.argwhere(~ok)[:4], got[~ok][:4], want[~ok][:4])


SHAPES = [(1, 1), (2, 31), (9, 33), (3, 127), (17, 128), (8, 129), (5, 255), (33, 300)]


@pytest.mark.parametrize("rows,cols", SHAPES)
def test_output_fields_equal_numpy(cuda_device, rows, cols):
    from hybrid_flood_b200 import output

    s, mask, _, st, rng = _case(rows, cols, rows * cols)
    odd = np.asarray([0.0, -0.0, 1e-42, -3e-39, 1e-30, 7e-20, 3e38, -2e38, 1e20, np.inf, np.nan], f4)
    at = rng.random((rows, cols)) < 0.3
    st[1][at] = rng.choice(odd, int(at.sum()))
    st[2][at] = rng.choice(odd, int(at.sum()))
    st[0][rng.random((rows, cols)) < 0.05] = 3e30
    dry = f4(s.params.dry_tolerance)
    fields = output.output_fields(s, _dev(st))
    fields = list(fields.values()) if isinstance(fields, dict) else list(fields)
    with np.errstate(all="ignore"):
        wet = st[0] > dry
        u = np.where(wet, st[1] / np.where(wet, st[0], 1), f4(0)).astype(f4)
        v = np.where(wet, st[2] / np.where(wet, st[0], 1), f4(0)).astype(f4)
        speed = np.sqrt(u.astype(np.float64) ** 2 + v.astype(np.float64) ** 2).astype(f4)
    nan = f4(np.nan)
    for got, want in zip(fields, (st[0], u, v, speed)):
        _same(got, np.where(mask, want, nan).astype(f4))


@pytest.mark.parametrize("rows,cols", SHAPES)
@pytest.mark.parametrize("layout", ["reference6", "state5"])
@pytest.mark.parametrize("offset", [0, 1, 2])
def test_features_equal_numpy(cuda_device, rows, cols, layout, offset):
    import ctypes

    from hybrid_flood_b200 import _lib

    s, mask, bed, st, rng = _case(rows, cols, 3 * rows + cols)
    dry = f4(s.params.dry_tolerance)
    mean = np.asarray([0.1, 0.01, -0.02, 3.0, 5.0], f4)
    std = np.asarray([0.08, 0.2, 0.15, 4.0, 5.0], f4)
    terrain, rough = rng.normal(size=(2, rows, cols)).astype(f4)
    h, hu, hv = st
    rain = f4(0.7)
    if layout == "reference6":
        wet = h > dry
        den = np.maximum(h, dry)
        u, v = (np.where(wet, x / den, f4(0)).astype(f4) for x in (hu, hv))
        ch = [np.where(mask, (x - mean[q]) / std[q], f4(0)) for q, x in enumerate((h, u, v))]
        ch += [np.full_like(h, rain), terrain, rough]
    else:
        ch = [np.where(mask, (x - mean[q]) / std[q], f4(0))
              for q, x in enumerate((h, hu, hv, bed, np.full_like(h, rain)))]
    want = np.stack(ch, -1).astype(f4)
    state = _dev(st, pad=3)
    lib = _lib.load()
    pt, pr = torch.from_numpy(terrain).cuda(), torch.from_numpy(rough).cuda()
    for dtype in (torch.float32, torch.bfloat16):
        buf = torch.full((want.size + 8,), 9.0, device="cuda", dtype=dtype)
        out = buf[offset: offset + want.size]
        rc = lib.swe_network_features(
            s._handle, state.h.data_ptr(), state.hu.data_ptr(), state.hv.data_ptr(), state.h.stride(0),
            0 if layout == "reference6" else 1, mean.ctypes.data, std.ctypes.data,
            ctypes.c_float(rain), pt.data_ptr(), pr.data_ptr(), out.data_ptr(), int(dtype == torch.bfloat16),
            torch.cuda.current_stream().cuda_stream)
        assert rc == 0
        torch.cuda.synchronize()
        ref = torch.from_numpy(want.ravel()).to(dtype)
        assert torch.equal(out.cpu(), ref)
        assert bool((buf[:offset] == 9).all()) and bool((buf[offset + want.size:] == 9).all())


@pytest.mark.parametrize("rows,cols", SHAPES)
@pytest.mark.parametrize("channels,dtype", [(1, torch.float32), (3, torch.float32), (1, torch.bfloat16), (3, torch.bfloat16)])
def test_correction_equals_numpy(cuda_device, rows, cols, channels, dtype):
    from hybrid_flood_b200 import hybrid

    s, mask, _, st, rng = _case(rows, cols, 5 * rows + cols)
    st[0] = np.where(mask, st[0], f4(0))
    dry = f4(s.params.dry_tolerance)
    res = torch.from_numpy((rng.normal(size=(rows, cols, channels)) * 0.1).astype(f4)).to(dtype)
    res[..., 0] = 0.0
    lim, relax = f4(0.05), f4(0.25)
    got = hybrid.apply_residual_correction(s, _dev(st, pad=1), res.cuda(), correction_relaxation=0.25,
                                           clip_limits=[0.05] * channels)
    h, hu, hv = st
    wet = h > dry
    den = np.maximum(h, dry)
    u, v = (np.where(wet, x / den, f4(0)).astype(f4) for x in (hu, hv))
    if channels == 3:
        r = np.clip(res.float().numpy(), -lim, lim)
        u, v = (u + relax * r[..., 1]).astype(f4), (v + relax * r[..., 2]).astype(f4)
    wet = mask & (h > dry)
    _same(got.h, h)
    _same(got.hu, np.where(wet, h * u, f4(0)).astype(f4))
    _same(got.hv, np.where(wet, h * v, f4(0)).astype(f4))
