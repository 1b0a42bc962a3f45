"""Speeds whose float64 root lies next to a tie of its rounding to float32.

``hypot(u, v)`` is the float64 root of u^2 + v^2 rounded to float32.  Where u^2 + v^2 is
the float64 next to m^2, m the midpoint of two float32, the root lies within a
few parts in 2^k of the tie between m and its neighbour, and a root that is off by
less than a float64 rounding can already give the other float32.  Such pairs are
searched for here; every one of them has to give NumPy's value.
"""

from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _pairs(side: int, count: int, seed: int) -> np.ndarray:
    """Float32 pairs (a, b) with float64(a^2 + b^2) one unit from m^2: m just above 1 (side 0) or below 2 (1)."""
    rng = np.random.default_rng(seed)
    found, n = [], 0
    while n < count:
        j = rng.integers(0, 1 << 15, 1 << 21).astype(np.float64)
        m = 1.0 + (2 * j + 1) * 2.0**-24 if side == 0 else 2.0 - (2 * j + 1) * 2.0**-24
        s = np.nextafter(m * m, rng.choice([0.0, 8.0], m.size))
        a = (m - rng.integers(1, 1 << 13, m.size) * 2.0**-24).astype(np.float32)
        r = s - a.astype(np.float64) ** 2
        b = np.sqrt(r).astype(np.float32)
        hit = a.astype(np.float64) ** 2 + b.astype(np.float64) ** 2 == s
        found.append(np.stack([a[hit], b[hit]]))
        n += int(hit.sum())
    return np.concatenate(found, axis=1)


@pytest.mark.parametrize("side", [0, 1])
def test_speed_next_to_a_tie(cuda_device, side):
    from hybrid_flood_b200.output import output_fields
    from hybrid_flood_b200.solver import B200ShallowWaterSolver

    p = _pairs(side, 400, 5 + side)
    p = np.concatenate([p, p[::-1], p * np.float32(2.0**-9), p * np.float32(0.5)], axis=1)
    a, b = (np.ascontiguousarray(x[None]) for x in p)
    s = B200ShallowWaterSolver(np.zeros_like(a), np.full_like(a, 0.03), np.ones(a.shape, bool), resolution_m=2.0,
                               rainfall_times_s=[0, 1], rainfall_rates_m_s=[0, 0])
    st = [torch.ones(a.shape, device="cuda"), torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda()]
    got = output_fields(s, st)["velocity"].cpu().numpy()
    want = np.sqrt(a.astype(np.float64) ** 2 + b.astype(np.float64) ** 2).astype(np.float32)
    assert np.array_equal(got, want), int((got != want).sum())
