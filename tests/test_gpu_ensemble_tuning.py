"""Tuning a small batch, or setting the rows it reports, keeps the split of its marches.

A batch of two 200 x 200 members marches a few rows a warp by default and 32 when it is
not split, which takes almost four times as long; twice the default's time tells
the two apart.
"""

from __future__ import annotations

import json

import pytest
import torch

from test_gpu_ensemble_split import _member

pytestmark = pytest.mark.gpu

SHAPES = [(200, 200)] * 2


def _ensemble(arithmetic="fast"):
    from hybrid_flood_b200.ensemble import B200Ensemble

    return B200Ensemble([_member(r, c, 7 + i, False)[0] for i, (r, c) in enumerate(SHAPES)], arithmetic=arithmetic)


def _states(shapes=SHAPES, masked=False):
    from hybrid_flood_b200.solver import SWEState

    return [SWEState(*(torch.from_numpy(a).cuda() for a in _member(r, c, 7 + i, masked)[1]))
            for i, (r, c) in enumerate(shapes)]


def _step_time(ens) -> float:
    ens.set_timing(True)
    ens.advance_(_states(), 100)
    times = []
    for _ in range(5):
        ens.advance_(_states(), 100)
        ms, n = ens.last_step_time()
        times.append(ms / n)
    return sorted(times)[2]


def test_autotune_keeps_the_split(cuda_device, tmp_path):
    ens = _ensemble()
    default = _step_time(ens)
    cache = tmp_path / "tune.json"
    best = ens.autotune(_states(), cache=cache)
    assert best == ens.rows_per_warp == json.loads(cache.read_text())[ens.shape_key()]["rows_per_warp"]
    assert _step_time(ens) < 2 * default
    again = _ensemble()
    assert again.autotune(_states(), cache=cache) == best  # from the cache
    assert _step_time(again) < 2 * default


def test_setting_the_rows_it_reports_keeps_the_split(cuda_device):
    ens = _ensemble()
    default = _step_time(ens)
    rows = ens.rows_per_warp
    ens.set_rows_per_warp(rows)
    assert _step_time(ens) < 2 * default
    ens.set_rows_per_warp(64)
    assert _step_time(ens) > 2 * default
    ens.set_rows_per_warp(rows)
    assert ens.rows_per_warp == rows and _step_time(ens) < 2 * default


def test_entries_of_another_plan_are_not_reused(cuda_device, tmp_path):
    """A winner cached when 32 rows meant an unsplit march (the key then had no plan) is timed anew."""
    import hashlib

    ens = _ensemble()
    old = hashlib.sha1(json.dumps({"shapes": sorted(ens.shapes), "arith": ens.arithmetic,
                                   "device": torch.cuda.get_device_name(ens.device)}).encode()).hexdigest()[:16]
    cache = tmp_path / "tune.json"
    cache.write_text(json.dumps({old: {"rows_per_warp": 256, "ms_per_step": {}}}))
    default = _step_time(ens)
    ens.autotune(_states(), cache=cache)
    assert _step_time(ens) < 2 * default


@pytest.mark.parametrize("shapes", [[(1, 1)], [(31, 64)], [(33, 63)], [(34, 130)], [(200, 200)] * 2, [(130, 1000)] * 3,
                                    [(512, 512)] * 4, [(400, 400)] * 9, [(5, 300), (97, 33), (256, 256)]], ids=str)
@pytest.mark.parametrize("masked", [False, True])
@pytest.mark.parametrize("arithmetic", ["fast", "exact"])
def test_split_equals_forced_32_rows(cuda_device, monkeypatch, shapes, masked, arithmetic):
    from hybrid_flood_b200.ensemble import B200Ensemble

    members = [_member(r, c, 7 + i, masked)[0] for i, (r, c) in enumerate(shapes)]
    got = []
    for rows in (None, "32"):
        if rows:
            monkeypatch.setenv("SWE_ENSEMBLE_ROWS", rows)
        ens = B200Ensemble(members, arithmetic=arithmetic)
        assert ens.rows_per_warp == 32
        cur = _states(shapes, masked)
        got.append((cur, [r[:2] for r in ens.advance_(cur, 9)]))
    assert got[0][1] == got[1][1]
    for x, y in zip(got[0][0], got[1][0]):
        for p, q in zip(x, y):
            assert torch.equal(p, q)
