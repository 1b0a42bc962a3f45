"""A small batch's marches are split below 32 rows: the results are the 32-row ones.

Fast arithmetic, where a march's first face is not rounded as its later ones are:
the split leads in with two dropped rows, so every bit has to be the same.
"""

from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _member(rows, cols, seed, masked):
    rng = np.random.default_rng(seed)
    f = lambda a: np.asarray(a, np.float32)  # noqa: E731
    mask = rng.random((rows, cols)) < 0.9 if masked else np.ones((rows, cols), bool)
    m = dict(bed=f(rng.uniform(0, 0.3, (rows, cols))), manning_n=f(np.full((rows, cols), 0.03)), domain_mask=mask,
             resolution_m=2.0, rainfall_times_s=f([0, 600]), rainfall_rates_m_s=f([1e-4, 2e-4]),
             boundary=(0, 1, 1, 0) if seed % 2 else (1, 1, 1, 1))
    h = np.where(mask, rng.uniform(0, 1, (rows, cols)) * (rng.random((rows, cols)) < 0.8), 0)
    return m, [f(h), f(h * rng.normal(0, 1, h.shape)), f(h * rng.normal(0, 1, h.shape))]


# One member to many, so that the split is 2, 4, 8 and 16 rows; heights around the 32-row
# seams; widths around a 64-column strip; one row; a batch that mixes shapes.
@pytest.mark.parametrize("shapes", [
    [(1, 1)], [(31, 64)], [(32, 65)], [(33, 63)], [(34, 130)], [(200, 200)] * 2, [(130, 1000)] * 3,
    [(512, 512)] * 4, [(400, 400)] * 9, [(5, 300), (97, 33), (256, 256)]], ids=str)
@pytest.mark.parametrize("masked", [False, True])
@pytest.mark.parametrize("arithmetic", ["fast", "exact"])
def test_split_marches_give_the_32_row_results(cuda_device, shapes, masked, arithmetic):
    from hybrid_flood_b200.ensemble import B200Ensemble
    from hybrid_flood_b200.solver import SWEState

    made = [_member(r, c, 7 + i, masked) for i, (r, c) in enumerate(shapes)]
    got = []
    for rows in (None, 32):
        ens = B200Ensemble([m for m, _ in made], arithmetic=arithmetic)
        if rows:
            ens.set_rows_per_warp(rows)
        cur = [SWEState(*(torch.from_numpy(a).cuda() for a in st)) for _, st in made]
        res = ens.advance_(cur, 9)
        got.append((cur, res))
    (a, ra), (b, rb) = got
    for x, y in zip(a, b):
        for p, q in zip(x, y):
            assert torch.equal(p, q)
    for (ta, na, la), (tb, nb, lb) in zip(ra, rb):
        assert ta == tb and na == nb
        # The volumes are float32 partials of a march, at most 32 rows of 2 columns a lane,
        # summed in float64: each is within 64 roundings of 2^-24 of the terms it adds.
        for k in la:
            assert la[k] == pytest.approx(lb[k], rel=64 * 2.0**-24, abs=64 * 2.0**-24 * abs(la["volume0"]))
