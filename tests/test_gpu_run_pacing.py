"""Runs to a known end time, whose launches are paced by the steps expected to be left.

A run of `advance_to_` reports the dt of every step.  Whatever was queued, the
steps taken end at the target, as many as a second run with that cap takes, and
the state is that of single steps with the logged dts (exact arithmetic, so bit
for bit).  The targets give runs shorter and longer than the first chunks (4 and
8 steps) and than one graph (32 or 50).
"""

from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _made(rows=70, cols=130, seed=4):
    rng = np.random.default_rng(seed)
    f = lambda a: np.asarray(a, np.float32)  # noqa: E731
    m = dict(bed=f(rng.uniform(0, 0.3, (rows, cols))), manning_n=f(np.full((rows, cols), 0.03)),
             domain_mask=np.ones((rows, cols), bool), resolution_m=2.0, rainfall_times_s=f([0, 600]),
             rainfall_rates_m_s=f([1e-5, 2e-5]), boundary=(0, 1, 1, 0))
    h = rng.uniform(0.2, 1, (rows, cols))
    return m, [f(h), f(h * rng.normal(0, 1, h.shape)), f(h * rng.normal(0, 1, h.shape))]


def _dev(st):
    from hybrid_flood_b200.solver import SWEState

    return SWEState(*(torch.from_numpy(a).cuda() for a in st))


def _solver(m):
    from hybrid_flood_b200.solver import B200ShallowWaterSolver

    kw = {k: v for k, v in m.items() if k not in ("bed", "manning_n", "domain_mask")}
    return B200ShallowWaterSolver(m["bed"], m["manning_n"], m["domain_mask"], **kw)


@pytest.mark.parametrize("target", [1e-4, 0.3, 0.8, 1.0, 4.0, 9.0, 20.0])
@pytest.mark.parametrize("batch", [False, True])
def test_paced_run_takes_the_steps_it_logs(cuda_device, target, batch):
    from hybrid_flood_b200.ensemble import B200Ensemble

    m, st = _made()
    s, cap = _solver(m), 2000
    log = torch.full((cap,), -1.0, dtype=torch.float64, device="cuda")
    if batch:
        run = lambda x, n: B200Ensemble([m], arithmetic="exact").advance_to_([x], 0.0, target, n, [log])[0]  # noqa: E731
    else:
        run = lambda x, n: s.advance_to_(x, 0.0, target, n, log)  # noqa: E731
    a = _dev(st)
    t, steps, _ = run(a, cap)
    dts = log.cpu().numpy()
    assert t == target and 1 <= steps < cap
    assert (dts[:steps] > 0).all() and (dts[steps:] == -1).all()
    b, clock = _dev(st), 0.0
    for dt in dts[:steps]:
        b, clock = s.step(b, float(dt), clock), clock + float(dt)
    assert clock == pytest.approx(target, rel=1e-15)
    for x, y in zip(a, b):
        assert torch.equal(x, y)
    # The cap at, and one step below, the number of steps needed.
    c = _dev(st)
    assert run(c, steps)[:2] == (target, steps)
    assert all(torch.equal(x, y) for x, y in zip(a, c))
    if steps > 1:
        short = run(_dev(st), steps - 1)
        assert short[1] == steps - 1 and short[0] < target


def test_outputs_close_together_and_far_apart(cuda_device):
    """Outputs between steps add steps that the pace has to count; device and host runs agree."""
    m, st = _made(33, 65, 5)
    times = np.asarray([0, 0.01, 0.02, 0.021, 5.0, 5.001, 5.002, 12.0], np.float32)
    s = _solver(m)
    a, b = s.run(_dev(st), times), s.run_to_host(st, times)
    assert a.steps_used == b.steps_used and a.outputs_written == b.outputs_written == len(times)
    for x, y in zip(a.states, b.states):
        assert np.array_equal(x.cpu().numpy(), np.asarray(y))
    # The same outputs by runs that each end at one: at most a rounding of the clock apart.
    x, steps = _dev(st), 0
    for i in range(1, len(times)):
        steps += s.advance_to_(x, float(times[i - 1]), float(times[i]), 2000)[1]
        d = (a.states.h[i] - x.h).double().norm() / x.h.double().norm()
        assert float(d) < 1e-5
    assert abs(steps - a.steps_used) <= len(times)
