"""Start and end of runs for one domain and for batches of domains.

Exact arithmetic throughout: a member of a batch has to equal the same run alone
bit for bit, whatever its place in the batch (a launch takes 32 domains), and the
CFL maximum NumPy's.
"""

from __future__ import annotations

import numpy as np
import pytest
import torch

from oracle import swe_numpy as O

pytestmark = pytest.mark.gpu


def _member(rows, cols, seed, masked=False):
    rng = np.random.default_rng(seed)
    f = lambda a: np.asarray(a, np.float32)  # noqa: E731
    mask = rng.random((rows, cols)) < 0.9 if masked else np.ones((rows, cols), bool)
    m = dict(bed=f(rng.uniform(0, 0.3, (rows, cols))), manning_n=f(np.full((rows, cols), 0.03)), domain_mask=mask,
             resolution_m=2.0, rainfall_times_s=f([0, 600]), rainfall_rates_m_s=f([1e-5, 2e-5]), boundary=(0, 1, 1, 0))
    h = np.where(mask, rng.uniform(0, 1, (rows, cols)) * (rng.random((rows, cols)) < 0.8), 0)
    return m, [f(h), f(h * rng.normal(0, 1, h.shape)), f(h * rng.normal(0, 1, h.shape))]


def _solver(m):
    from hybrid_flood_b200.solver import B200ShallowWaterSolver

    kw = {k: v for k, v in m.items() if k not in ("bed", "manning_n", "domain_mask")}
    return B200ShallowWaterSolver(m["bed"], m["manning_n"], m["domain_mask"], **kw)


def _dev(st):
    from hybrid_flood_b200.solver import SWEState

    return SWEState(*(torch.from_numpy(a).cuda() for a in st))


@pytest.mark.parametrize("n", [1, 31, 32, 33, 65])
def test_members_of_a_batch_equal_single_runs(cuda_device, n):
    from hybrid_flood_b200.ensemble import B200Ensemble

    shapes = [(1, 1), (5, 64), (9, 65), (40, 130), (70, 63), (33, 191)]
    made = [_member(*shapes[m % len(shapes)], 50 + m, masked=m % 3 == 0) for m in range(n)]
    ens = B200Ensemble([m for m, _ in made], arithmetic="exact")
    cur = [_dev(st) for _, st in made]
    res = ens.advance_(cur, 3, [10.0 * m for m in range(n)])
    for i in sorted({0, n // 2, n - 1, max(0, n - 2)}):
        s = _solver(made[i][0])
        one, t, steps, ledger = s.advance(_dev(made[i][1]), 3, 10.0 * i)
        assert res[i][0] == t and res[i][1] == steps == 3
        for a, b in zip(cur[i], one):
            assert torch.equal(a, b)
        # The start's own ledger term; the step's terms are float partials of a march's
        # rows, and the two marches differ in height.
        assert res[i][2]["volume0"] == pytest.approx(ledger["volume0"], rel=1e-12, abs=1e-12)


@pytest.mark.parametrize("rows,cols", [(1, 1), (2, 127), (3, 129), (500, 300), (1030, 77), (40, 4100)])
@pytest.mark.parametrize("masked", [False, True])
def test_cfl_maximum_and_volume_equal_numpy(cuda_device, rows, cols, masked):
    m, st = _member(rows, cols, rows + cols, masked)
    s = _solver(m)
    p = O.make_params(m["bed"], m["manning_n"], m["domain_mask"],
                      **{k: v for k, v in m.items() if k not in ("bed", "manning_n", "domain_mask")})
    for pad in (0, 3):
        wide = []
        for a in st:
            w = torch.zeros((rows, cols + pad), device="cuda")
            w[:, :cols] = torch.from_numpy(a)
            wide.append(w[:, :cols])
        assert s.max_inverse_dt(wide) == float(O.max_inverse_dt(O.State(*st), p))
    _, _, _, ledger = s.advance(_dev(st), 0)
    want = float(np.where(m["domain_mask"], st[0], 0).astype(np.float64).sum()) * 4.0
    assert ledger["volume0"] == pytest.approx(want, rel=1e-12)


@pytest.mark.parametrize("value", [np.nan, np.inf])
def test_non_finite_start_is_reported(cuda_device, value):
    m, st = _member(40, 70, 3)
    st[0][17, 5] = value
    with pytest.raises(RuntimeError):
        _solver(m).advance(_dev(st), 4)


def test_state_is_returned_through_any_pitch(cuda_device):
    m, st = _member(37, 65, 9)
    s = _solver(m)
    want, *_ = s.advance(_dev(st), 5)
    wide = torch.full((3, 37, 80), 7.0, device="cuda")
    from hybrid_flood_b200.solver import SWEState

    view = SWEState(*(wide[q, :, :65] for q in range(3)))
    for v, a in zip(view, st):
        v.copy_(torch.from_numpy(a))
    s.advance_(view, 5)
    for v, w in zip(view, want):
        assert torch.equal(v, w)
    assert bool((wide[:, :, 65:] == 7.0).all())
