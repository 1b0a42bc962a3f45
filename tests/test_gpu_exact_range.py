"""Exact arithmetic outside the range of its branch-free form.

Domains whose controls lie outside it (a dry tolerance below 2^-30, a gravity or cell size out
of the ordinary) run the IEEE operations throughout, other domains for the rows whose cells
leave it.  Both are compared, bit for bit, with the one-cell-per-lane kernel, which has
the IEEE operations only.
"""

from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _member(rows, cols, seed, masked=False, depth=1.0, speed=1.0, **controls):
    rng = np.random.default_rng(seed)
    f = lambda a: np.asarray(a, np.float32)  # noqa: E731
    mask = rng.random((rows, cols)) < 0.9 if masked else np.ones((rows, cols), bool)
    m = dict(bed=f(rng.uniform(0, 0.3, (rows, cols))), manning_n=f(np.full((rows, cols), 0.03)), domain_mask=mask,
             resolution_m=2.0, rainfall_times_s=f([0, 600]), rainfall_rates_m_s=f([1e-5, 2e-5]), boundary=(0, 1, 1, 0))
    m.update(controls)
    h = np.where(mask, rng.uniform(0, depth, (rows, cols)) * (rng.random((rows, cols)) < 0.8), 0)
    u = rng.normal(0, speed, (2, rows, cols))
    return m, [f(h), f(h * u[0]), f(h * u[1])]


def _solver(m):
    from hybrid_flood_b200.solver import B200ShallowWaterSolver

    kw = {k: v for k, v in m.items() if k not in ("bed", "manning_n", "domain_mask")}
    return B200ShallowWaterSolver(m["bed"], m["manning_n"], m["domain_mask"], arithmetic="exact", **kw)


def _dev(st):
    from hybrid_flood_b200.solver import SWEState

    return SWEState(*(torch.from_numpy(a).cuda() for a in st))


def _step_us(m, st, steps=64):
    s = _solver(m)
    s.resident_load(_dev(st))
    s.resident_steps(steps)
    e0, e1 = (torch.cuda.Event(enable_timing=True) for _ in range(2))
    times = []
    for _ in range(5):
        e0.record()
        s.resident_steps(steps)
        e1.record()
        torch.cuda.synchronize()
        times.append(e0.elapsed_time(e1) / steps * 1e3)
    return sorted(times)[2]


OUTSIDE = [dict(dry_tolerance_m=0.0), dict(dry_tolerance_m=1e-12), dict(dry_tolerance_m=2.0), dict(gravity_m_s2=0.01),
           dict(gravity_m_s2=100.0), dict(resolution_m=2.0e5), dict(resolution_m=5.0e-4)]


@pytest.mark.parametrize("controls", OUTSIDE, ids=str)
@pytest.mark.parametrize("rows,cols,masked", [(1, 1, False), (33, 65, False), (40, 130, True), (70, 257, False)])
def test_domains_outside_the_range(cuda_device, monkeypatch, controls, rows, cols, masked):
    m, st = _member(rows, cols, 3, masked, depth=3.0, **controls)
    s, a = _solver(m), _dev(st)
    ra = s.advance_(a, 15)
    one = s.step(_dev(st), 0.01, 3.0)
    monkeypatch.setenv("SWE_RUN_VEC", "1")
    t, b = _solver(m), _dev(st)
    rb = t.advance_(b, 15)
    assert ra[:2] == rb[:2]
    for x, y in zip(a, b):
        assert torch.equal(x, y)
    wide = [torch.zeros((rows, cols + 1 + cols % 2), device="cuda") for _ in range(3)]
    for w, v in zip(wide, st):
        w[:, :cols] = torch.from_numpy(v)
    for x, y in zip(one, s.step([w[:, :cols] for w in wide], 0.01, 3.0)):  # an odd pitch: one cell per lane
        assert torch.equal(x, y)


@pytest.mark.parametrize("masked", [False, True])
@pytest.mark.parametrize("table", ["1", "0"])
def test_batch_with_members_on_both_sides(cuda_device, monkeypatch, masked, table):
    from hybrid_flood_b200.ensemble import B200Ensemble

    monkeypatch.setenv("SWE_ENS_PARAM_TABLE", table)
    made = [_member(40 + 30 * i, 65 + 64 * i, i, masked, **c) for i, c in enumerate([{}, OUTSIDE[0], OUTSIDE[3]])]
    states = [_dev(st) for _, st in made]
    res = B200Ensemble([m for m, _ in made], arithmetic="exact").advance_(states, 13)
    for (m, st), got, r in zip(made, states, res):
        want = _dev(st)
        assert _solver(m).advance_(want, 13)[:2] == r[:2]
        for x, y in zip(got, want):
            assert torch.equal(x, y)


def test_domain_outside_the_range_evaluates_its_rows_once(cuda_device):
    """On a flowing state a step of IEEE operations takes 1.6 times the branch-free one (1024^2: 37 and 23 us);
    with both evaluated, and the IEEE operations as calls, it took 2.7 times (63 us)."""
    m, st = _member(1024, 1024, 3)
    assert _step_us({**m, "dry_tolerance_m": 0.0}, st) < 2.1 * _step_us(m, st)


@pytest.mark.parametrize("masked", [False, True])
def test_deep_water_stays_in_the_range(cuda_device, masked):
    """A grid 2000 m deep takes the branch-free form: the same time as a shallow one (three times before)."""
    m, st = _member(1024, 1024, 5, masked)
    deep = [np.where(m["domain_mask"], st[0] + np.float32(2000), 0).astype(np.float32), *st[1:]]
    assert _step_us(m, deep) < 1.5 * _step_us(m, st)


@pytest.mark.parametrize("depth,speed", [(4000.0, 30.0), (9.0e4, 1.0), (1.0, 9.0e4), (3.0e4, 3.0e4), (1.0e6, 1.0e6)])
@pytest.mark.parametrize("masked", [False, True])
def test_rows_below_and_above_the_limit(cuda_device, monkeypatch, depth, speed, masked):
    """Runs and steps whose rows lie on both sides of 65536 m or m/s, and cross it."""
    m, st = _member(70, 200, 9, masked)
    big, big_st = _member(70, 200, 11, masked, depth=depth, speed=speed)
    big["domain_mask"] = m["domain_mask"]
    pick = (np.arange(70) // 9 % 3 == 1)[:, None] & m["domain_mask"]
    st = [np.where(pick, b, a).astype(np.float32) for a, b in zip(st, big_st)]
    s, a = _solver(m), _dev(st)
    ra = s.advance_(a, 25)
    dt = 0.1 / (depth + speed)
    one = s.step(_dev(st), dt, 3.0)
    monkeypatch.setenv("SWE_RUN_VEC", "1")
    b = _dev(st)
    assert _solver(m).advance_(b, 25)[:2] == ra[:2]
    for x, y in zip(a, b):
        assert torch.equal(x, y)
    wide = [torch.zeros((70, 201), device="cuda") for _ in range(3)]
    for w, v in zip(wide, st):
        w[:, :200] = torch.from_numpy(v)
    for x, y in zip(one, s.step([w[:, :200] for w in wide], dt, 3.0)):
        assert torch.equal(x, y)


def test_large_depths_and_speeds_equal_numpy(cuda_device):
    """Without friction every operation of the step is one IEEE operation of the reference."""
    from oracle import swe_numpy as O

    for depth, speed in ((3.0e4, 50.0), (50.0, 3.0e4), (6.0e4, 6.0e4), (2.0e5, 1.0e5)):
        m, st = _member(40, 150, 13, depth=depth, speed=speed, manning_n=np.zeros((40, 150), np.float32))
        got = _solver(m).step(_dev(st), 0.01, 33.0)
        kw = {k: v for k, v in m.items() if k not in ("bed", "manning_n", "domain_mask")}
        want = O.finite_volume_step(O.State(*st), O.make_params(m["bed"], m["manning_n"], m["domain_mask"], **kw), 0.01,
                                    33.0)
        for g, w in zip(got, want):
            assert np.array_equal(g.cpu().numpy(), w)
