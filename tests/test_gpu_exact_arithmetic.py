"""The branch-free exact arithmetic of the step against NumPy, bit for bit.

With n = 0 the friction term is exactly 1 + 0, so every operation of the step
is one IEEE float32 operation of the reference and the results have to be
equal (``np.array_equal``), whichever form computed a row: the branch-free one,
or the IEEE operations that rows outside its range take (depths or speeds of
1024 and more, infinities, NaN).  States that overflow are compared with the
one-cell-per-lane kernel instead, which uses the IEEE operations throughout
(its maxima drop a NaN where NumPy's keep it).  With friction the power differs from NumPy's
by at most an ulp, which the update passes on at most once: 2e-6 relative, the
bound of the one-step parity test.
"""

from __future__ import annotations

import numpy as np
import pytest
import torch

from oracle import swe_numpy as O

pytestmark = pytest.mark.gpu


def _case(rows, cols, dx, seed, *, depth=1.0, speed=1.0, n=0.0, masked=False, dry=1.0e-3, steps_z=0.5):
    rng = np.random.default_rng(seed)
    f = lambda a: np.asarray(a, np.float32)  # noqa: E731
    bed = f(rng.uniform(-steps_z, steps_z, (rows, cols)) * (rng.random((rows, cols)) < 0.7))
    h = rng.uniform(0.0, depth, (rows, cols)) * (rng.random((rows, cols)) < 0.85)
    h = f(h * 10.0 ** -(rng.uniform(0, 6, (rows, cols)) ** 2 / 6))
    u = rng.normal(0, speed, (2, rows, cols)) * 10.0 ** -(rng.uniform(0, 6, (2, rows, cols)) ** 2 / 4)
    u *= rng.random((2, rows, cols)) < 0.8
    mask = rng.random((rows, cols)) < 0.9 if masked else np.ones((rows, cols), bool)
    h = f(np.where(mask, h, 0))
    kw = dict(resolution_m=dx, rainfall_times_s=f([0, 60, 600]), rainfall_rates_m_s=f([0, 2e-5, 1e-5]),
              boundary=(0, 1, 1, 0), cfl=0.45, dry_tolerance_m=dry, max_dt_s=10.0)
    return (bed, np.full((rows, cols), n, np.float32), mask), kw, (h, f(h * u[0].astype(np.float32)),
                                                                   f(h * u[1].astype(np.float32)))


def _both(fields, kw, state, dt=0.037, t=33.0):
    from hybrid_flood_b200.solver import B200ShallowWaterSolver

    s = B200ShallowWaterSolver(*fields, **kw, arithmetic="exact")
    got = [a.cpu().numpy() for a in s.step([torch.from_numpy(a).cuda() for a in state], dt, t)]
    with np.errstate(all="ignore"):
        p = O.make_params(*fields, **kw)
        want = O.finite_volume_step(O.State(*state), p, dt, t)
    return s, got, want


def _ieee(s, state, dt=0.037, t=33.0):
    """The same step by the one-cell-per-lane kernel (an odd row pitch selects it)."""
    wide = []
    for a in state:
        w = torch.zeros((a.shape[0], a.shape[1] + 1 + a.shape[1] % 2), device="cuda")
        w[:, : a.shape[1]] = torch.from_numpy(a)
        wide.append(w[:, : a.shape[1]])
    assert wide[0].stride(0) % 2 == 1
    return [a.cpu().numpy() for a in s.step(wide, dt, t)]


@pytest.mark.parametrize("rows,cols", [(1, 1), (3, 63), (9, 64), (33, 65), (70, 200)])
@pytest.mark.parametrize("dx,masked", [(2.0, False), (10.0, False), (3.7, True)])
def test_frictionless_step_equals_numpy(cuda_device, rows, cols, dx, masked):
    fields, kw, st = _case(rows, cols, dx, rows * 1000 + cols, masked=masked)
    s, got, want = _both(fields, kw, st)
    for g, w in zip(got, want):
        assert np.array_equal(g, w)
    dt = s.cfl_dt([torch.from_numpy(a).cuda() for a in st])
    assert dt == O.compute_cfl_dt(O.State(*st), O.make_params(*fields, **kw))


@pytest.mark.parametrize("depth,speed,dry", [(900.0, 30.0, 1e-3), (5000.0, 1.0, 1e-3), (1.0, 4000.0, 1e-3),
                                             (1.0, 1e-25, 1e-3), (1.0, 1.0, 0.0), (1.0, 1.0, 1e-12)])
def test_frictionless_step_at_the_ends_of_the_range(cuda_device, depth, speed, dry):
    """Depths and speeds on both sides of the limit, vanishing momenta, dry tolerances outside the range."""
    fields, kw, st = _case(40, 150, 10.0, 7, depth=depth, speed=speed, dry=dry)
    s, got, want = _both(fields, kw, st)
    if dry > 0:
        for g, w in zip(got, want):
            assert np.array_equal(g, w)
    for g, w in zip(got, _ieee(s, st)):
        assert np.array_equal(g, w, equal_nan=True)


@pytest.mark.parametrize("where", [(0, 0), (17, 63), (20, 64), (39, 149)])
@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan, 3.0e38, 1.0e20])
@pytest.mark.parametrize("field", [0, 1])
def test_non_finite_and_huge_cells(cuda_device, where, value, field):
    fields, kw, st = _case(40, 150, 2.0, 11)
    st[field][where] = abs(value) if field == 0 else value
    s, got, _ = _both(fields, kw, st)
    for g, w in zip(got, _ieee(s, st)):
        assert np.array_equal(g, w, equal_nan=True)


def test_every_mantissa_as_depth(cuda_device):
    """All 2^23 float mantissas as depths (velocities divide by each of them, roots and wave speeds follow)."""
    rng = np.random.default_rng(3)
    rows, cols = 2048, 4096
    m = rng.permutation(np.arange(1 << 23, dtype=np.uint32)).reshape(rows, cols)
    h = ((np.uint32(126) << np.uint32(23)) | m).view(np.float32)
    hu = (h * rng.normal(0, 0.5, h.shape).astype(np.float32)).astype(np.float32)
    hv = (h * rng.normal(0, 0.5, h.shape).astype(np.float32)).astype(np.float32)
    fields, kw, _ = _case(rows, cols, 10.0, 5)
    _, got, want = _both(fields, kw, (h, hu, hv), dt=0.2)
    for g, w in zip(got, want):
        assert np.array_equal(g, w)


@pytest.mark.parametrize("dx", [2.0, 10.0])
def test_step_with_friction(cuda_device, dx):
    fields, kw, st = _case(65, 130, dx, 21, n=0.05)
    _, got, want = _both(fields, kw, st)
    np.testing.assert_array_equal(got[0], want[0])
    for g, w in zip(got[1:], want[1:]):
        np.testing.assert_allclose(g, w, rtol=2e-6, atol=1e-12)


@pytest.mark.parametrize("masked", [False, True])
def test_run_rows_leave_and_enter_the_range(cuda_device, masked):
    """A run whose rows take both forms: CFL steps equal NumPy's in number, clock and state."""
    from hybrid_flood_b200.solver import B200ShallowWaterSolver

    fields, kw, st = _case(70, 130, 2.0, 31, masked=masked)
    st[0][30:34, 60:70] = np.where(fields[2][30:34, 60:70], 1100.0, 0.0)
    s = B200ShallowWaterSolver(*fields, **kw, arithmetic="exact")
    new, t, n, _ = s.advance([torch.from_numpy(a).cuda() for a in st], 12)
    p = O.make_params(*fields, **kw)
    ref, clock = O.State(*st), 0.0
    for _ in range(12):
        dt = O.compute_cfl_dt(ref, p)
        ref = O.finite_volume_step(ref, p, dt, clock)
        clock += dt
    assert n == 12 and t == clock
    for g, w in zip(new, ref):
        assert np.array_equal(g.cpu().numpy(), w)
