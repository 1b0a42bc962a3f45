"""An ``advance_`` that fails leaves the caller's state as it was."""

from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


# The run stops at once, or after a step that was taken: a depth whose square overflows has a
# finite wave speed, but its momentum flux is infinite, which the next step's maximum shows.
@pytest.mark.parametrize("value", [np.nan, np.inf, 1.0e30])
@pytest.mark.parametrize("shape", [(1, 1), (40, 130), (33, 257)], ids=str)
@pytest.mark.parametrize("arithmetic", ["fast", "exact"])
def test_failed_advance_keeps_the_state(cuda_device, shape, value, arithmetic):
    from hybrid_flood_b200.solver import B200ShallowWaterSolver, SWEState

    rng = np.random.default_rng(3)
    s = B200ShallowWaterSolver(np.zeros(shape, np.float32), np.full(shape, 0.03, np.float32), np.ones(shape, bool),
                               resolution_m=2.0, rainfall_times_s=[0, 600], rainfall_rates_m_s=[1e-5, 2e-5],
                               arithmetic=arithmetic)
    st = [rng.uniform(0.1, 1, shape).astype(np.float32) for _ in range(3)]
    st[0].flat[-1] = value
    pad = [torch.full((shape[0], shape[1] + 3), 7.0, device="cuda") for _ in range(3)]
    cur = SWEState(*(p[:, : shape[1]] for p in pad))
    for t, a in zip(cur, st):
        t.copy_(torch.from_numpy(a))
    before = [p.clone() for p in pad]
    with pytest.raises(RuntimeError, match="non-finite"):
        s.advance_(cur, 40)
    for p, q in zip(pad, before):
        assert torch.equal(p.view(torch.int32), q.view(torch.int32))
    # The solver goes on with the next state.
    good = SWEState(*(torch.from_numpy(np.minimum(np.nan_to_num(a, posinf=1.0), 1.0)).cuda() for a in st))
    assert s.advance_(good, 5)[1] == 5
