"""A single reverse step, whose update is rebuilt from the faces within the march.

On grids with marches of several rows and more than one wave of them, against the
two-kernel form that aliased buffers take: as in test_gpu_adjoint_march, 1e-5 of the
field's norm.  (The edges of strips and chunks are there.)
"""

from __future__ import annotations

import pytest
import torch

from conftest import rel_l2
from test_gpu_adjoint_march import _case, _reverse, _wide

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,cols", [(2, 2), (300, 420), (700, 901), (1025, 1024)])
@pytest.mark.parametrize("masked,bnd", [(False, (1, 1, 0, 0)), (True, (0, 1, 1, 0))])
@pytest.mark.parametrize("pad", [0, 3])
def test_faces_march_equals_the_two_kernel_form(cuda_device, rows, cols, masked, bnd, pad):
    s, st, lam = _case(rows, cols, masked, bnd, 7 * rows + cols)
    lam2 = [t.clone() for t in lam]
    want, gn, gr = _reverse(s, st, lam2, lam2)  # aliased: two kernels
    st, lam = [_wide(t, pad) for t in st], [_wide(t, pad) for t in lam]
    out = [_wide(torch.zeros(s.shape, device="cuda"), pad) for _ in range(3)]
    got, gn1, gr1 = _reverse(s, st, lam, out)
    for a, b in zip(got, want):
        assert rel_l2(a, b) <= 1e-5
    assert rel_l2(gn1, gn) <= 1e-5
    # A sum over the cells of terms of both signs, each within 1e-5: of the sum of magnitudes.
    assert gr1 == pytest.approx(gr, abs=1e-5 * 0.05 * 2e-5 * sum(float(t.abs().sum()) for t in lam))


def _time_us(fn, n=30):
    for _ in range(3):
        fn()
    e0, e1 = (torch.cuda.Event(enable_timing=True) for _ in range(2))
    times = []
    for _ in range(5):
        e0.record()
        for _ in range(n):
            fn()
        e1.record()
        torch.cuda.synchronize()
        times.append(e0.elapsed_time(e1) / n * 1e3)
    return sorted(times)[2]


def test_reverse_step_is_a_few_forward_steps(cuda_device):
    """At 2048^2 a reverse step takes 2.8 exact forward steps (208 and 75 us); 4.9 with the update of every
    cell rebuilt apart from its four faces."""
    from hybrid_flood_b200.adjoint import adjoint_step
    from hybrid_flood_b200.solver import SWEState

    s, st, lam = _case(2048, 2048, False, (0, 0, 0, 0), 3)
    gn, gr = torch.zeros(s.shape, device="cuda"), torch.zeros(1, dtype=torch.float64, device="cuda")
    state, lam = SWEState(*st), SWEState(*lam)
    reverse = _time_us(lambda: adjoint_step(s, state, lam, 0.05, 3.0, gn, gr))
    forward = _time_us(lambda: s.step(state, 0.05, 3.0))
    assert reverse < 3.8 * forward
