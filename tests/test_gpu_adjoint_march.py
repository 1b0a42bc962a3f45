"""The one-kernel reverse step against the two-kernel form that aliased buffers take.

Both evaluate the same derivative in float32, in pairs of cells and one cell at
a time: each value is a sum of about a hundred rounded terms with cancellations
of a factor of about a hundred, 100 x 100 x 6e-8 of the largest terms in the worst
case and their square root in the mean, so 1e-5 of the field's norm.
"""

from __future__ import annotations

import ctypes

import numpy as np
import pytest
import torch

from conftest import rel_l2

pytestmark = pytest.mark.gpu

SHAPES = [(1, 1), (1, 7), (5, 2), (3, 59), (4, 60), (6, 61), (9, 62), (17, 121), (33, 130), (70, 64)]


def _case(rows, cols, masked, bnd, seed):
    from hybrid_flood_b200.solver import B200ShallowWaterSolver

    rng = np.random.default_rng(seed)
    f = lambda a: np.asarray(a, np.float32)  # noqa: E731
    mask = rng.random((rows, cols)) < 0.85 if masked else np.ones((rows, cols), bool)
    bed = f(rng.uniform(0, 0.4, (rows, cols)))
    man = f(rng.uniform(0.02, 0.06, (rows, cols)))
    s = B200ShallowWaterSolver(bed, man, mask, resolution_m=2.0, rainfall_times_s=f([0, 100]),
                               rainfall_rates_m_s=f([1e-5, 2e-5]), boundary=bnd, dry_tolerance_m=1e-3)
    h = np.where(mask, rng.uniform(0.0, 1.0, (rows, cols)) * (rng.random((rows, cols)) < 0.9), 0)
    st = [f(h), f(h * rng.normal(0, 1.0, h.shape)), f(h * rng.normal(0, 1.0, h.shape))]
    lam = [f(rng.normal(0, 1, h.shape)) for _ in range(3)]
    return s, [torch.from_numpy(a).cuda() for a in st], [torch.from_numpy(a).cuda() for a in lam]


def _reverse(s, st, lam, out):
    """swe_adjoint_step into ``out`` (which may be ``lam`` itself): (lam_out, grad_n2, grad_rain)."""
    p = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
    gn = torch.full(s.shape, 0.25, device="cuda")
    gr = torch.zeros(1, dtype=torch.float64, device="cuda")
    rc = s._lib.swe_adjoint_step(s._handle, *(p(t) for t in st), st[0].stride(0), *(p(t) for t in lam),
                                 lam[0].stride(0), *(p(t) for t in out), out[0].stride(0), p(gn), p(gr), 0.05, 40.0,
                                 ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert rc == 0
    return [t.cpu().numpy() for t in out], gn.cpu().numpy(), float(gr)


def _wide(t, pad):
    w = torch.zeros((t.shape[0], t.shape[1] + pad), device="cuda")
    w[:, : t.shape[1]] = t
    return w[:, : t.shape[1]]


@pytest.mark.parametrize("rows,cols", SHAPES)
@pytest.mark.parametrize("masked,bnd", [(False, (0, 1, 0, 1)), (True, (1, 0, 1, 0))])
@pytest.mark.parametrize("pad", [0, 1])
def test_march_equals_the_two_kernel_form(cuda_device, rows, cols, masked, bnd, pad):
    s, st, lam = _case(rows, cols, masked, bnd, 100 * rows + cols)
    lam2 = [t.clone() for t in lam]
    want, gn, gr = _reverse(s, st, lam2, lam2)  # aliased: two kernels
    st, lam = [_wide(t, pad) for t in st], [_wide(t, pad) for t in lam]
    got, gn1, gr1 = _reverse(s, st, lam, [_wide(torch.zeros(s.shape, device="cuda"), pad) for _ in range(3)])
    for a, b in zip(got, want):
        assert rel_l2(a, b) <= 1e-5
    assert rel_l2(gn1, gn) <= 1e-5
    assert gr1 == pytest.approx(gr, rel=1e-5, abs=1e-12)


@pytest.mark.parametrize("rows,cols,masked", [(1, 3, False), (9, 61, True), (33, 130, False), (40, 127, True)])
def test_update_rebuilt_from_the_next_state(cuda_device, rows, cols, masked):
    """The rollout's reverse (which inverts the friction of its own output) against a chain of single
    reverse steps (which recompute the update).  The inversion loses up to the factor by which friction
    divides a momentum, 1000 at most: 1000 x 6e-8 at a cell, 1e-4 of the field."""
    from hybrid_flood_b200.adjoint import adjoint_step, gauge_rollout
    from hybrid_flood_b200.solver import SWEState

    s, st, _ = _case(rows, cols, masked, (0, 1, 0, 1), 7)
    n, dt = 6, 0.05
    man = torch.full(s.shape, 0.03, device="cuda", requires_grad=True)
    h0 = st[0].clone().requires_grad_(True)
    idx = torch.arange(min(8, rows * cols), device="cuda")
    obs = gauge_rollout(s, man, h0, 1.0, hu0=st[1], hv0=st[2], n_steps=n, dt=dt, gauge_index=idx, obs_every=n,
                        checkpoint_every=4)
    w = torch.linspace(0.5, 1.5, idx.numel(), device="cuda")[None]
    gn, gh = torch.autograd.grad(obs, (man, h0), w)
    states = [SWEState(*(t.clone() for t in st))]
    for k in range(n):
        states.append(s.step(states[-1], dt, k * dt))
    lam = SWEState(*(torch.zeros(s.shape, device="cuda") for _ in range(3)))
    lam.h.view(-1)[idx] += w[0]
    g2, gr = torch.zeros(s.shape, device="cuda"), torch.zeros(1, dtype=torch.float64, device="cuda")
    for k in range(n - 1, -1, -1):
        lam = adjoint_step(s, states[k], lam, dt, k * dt, g2, gr)
    assert rel_l2(gh.cpu().numpy(), lam.h.cpu().numpy()) <= 1e-4
    assert rel_l2(gn.cpu().numpy(), (g2 * 2 * man.detach()).cpu().numpy()) <= 1e-4
