"""Steps whose starts overlap (programmatic launch) against steps launched one after the other.

The same calls run in two processes, with ``SWE_PDL=0`` and ``SWE_PDL=1``; the overlap
must not show in a single bit of states, observations or gradients.  The rain-scale
gradient is a float64 sum in the order in which CTAs arrive, returned as a float32:
n additions in another order differ by at most n x 2^-53 of the sum of magnitudes
(n < 2^11 CTA terms here), far below a float32 rounding unless the terms cancel to
2^-18 of that sum, so the results are at most neighbouring floats: 2^-22.
"""

from __future__ import annotations

import os
import subprocess
import sys

import numpy as np
import pytest

from conftest import PKG_ROOT, REPO

pytestmark = pytest.mark.gpu

SCRIPT = r"""
import sys
import numpy as np, torch
from hybrid_flood_b200.adjoint import gauge_rollout
from hybrid_flood_b200.ensemble import B200Ensemble
from hybrid_flood_b200.solver import B200ShallowWaterSolver, SWEState

out = {}
f = lambda a: np.asarray(a, np.float32)


def member(rows, cols, seed, masked):
    rng = np.random.default_rng(seed)
    mask = rng.random((rows, cols)) < 0.9 if masked else np.ones((rows, cols), bool)
    m = dict(bed=f(rng.uniform(0, 0.3, (rows, cols))), manning_n=f(np.full((rows, cols), 0.03)), domain_mask=mask,
             resolution_m=2.0, rainfall_times_s=f([0, 600]), rainfall_rates_m_s=f([1e-4, 2e-4]), boundary=(0, 1, 1, 0))
    h = np.where(mask, rng.uniform(0, 1, (rows, cols)) * (rng.random((rows, cols)) < 0.8), 0)
    return m, [f(h), f(h * rng.normal(0, 1, h.shape)), f(h * rng.normal(0, 1, h.shape))]


def solver(m, arith):
    kw = {k: v for k, v in m.items() if k not in ("bed", "manning_n", "domain_mask")}
    return B200ShallowWaterSolver(m["bed"], m["manning_n"], m["domain_mask"], arithmetic=arith, **kw)


def dev(st):
    return SWEState(*(torch.from_numpy(a).cuda() for a in st))


def keep(name, tensors):
    for i, t in enumerate(tensors):
        out[f"{name}_{i}"] = t.detach().cpu().numpy()


for arith in ("fast", "exact"):
    for masked in (False, True):
        tag = f"{arith}_{masked}"
        for rows, cols in ((40, 130), (200, 511), (1000, 1030)):
            m, st = member(rows, cols, rows, masked)
            s = solver(m, arith)
            x = dev(st)
            s.advance_(x, 77)
            keep(f"advance_{tag}_{rows}", x)
            x = dev(st)
            s.advance_to_(x, 0.0, 3.0, 500)
            keep(f"advance_to_{tag}_{rows}", x)
        made = [member(r, c, r + c, masked) for r, c in ((97, 130), (64, 64), (301, 200))]
        ens = B200Ensemble([m for m, _ in made], arithmetic=arith)
        xs = [dev(st) for _, st in made]
        ens.advance_(xs, 60)
        ens.advance_to_(xs, 100.0, 104.0, 500)
        for i, x in enumerate(xs):
            keep(f"ensemble_{tag}_{i}", x)
        for rows, cols in ((40, 130), (301, 257)):
            m, st = member(rows, cols, rows, masked)
            s = solver(m, arith)
            man = torch.full(s.shape, 0.03, device="cuda", requires_grad=True)
            h0 = torch.from_numpy(st[0]).cuda().requires_grad_(True)
            rain = torch.tensor(1.0, dtype=torch.float64, device="cuda", requires_grad=True)
            idx = torch.arange(0, rows * cols, 17, device="cuda")
            obs = gauge_rollout(s, man, h0, rain, hu0=dev(st).hu, hv0=dev(st).hv, n_steps=12, dt=0.05, gauge_index=idx,
                                obs_every=4, checkpoint_every=5)
            gn, gh, gr = torch.autograd.grad(obs, (man, h0, rain), torch.ones_like(obs))
            keep(f"gauge_{tag}_{rows}", (obs, gn, gh))
            out[f"rain_{tag}_{rows}"] = gr.detach().cpu().numpy()
np.savez(sys.argv[1], **out)
"""


def test_overlapped_steps_equal_sequential_ones(cuda_device, tmp_path):
    got = []
    for pdl in ("0", "1"):
        env = {**os.environ, "SWE_PDL": pdl, "PYTHONPATH": os.pathsep.join([str(PKG_ROOT), str(REPO)])}
        path = tmp_path / f"pdl{pdl}.npz"
        r = subprocess.run([sys.executable, "-c", SCRIPT, str(path)], env=env, capture_output=True, text=True, timeout=600)
        assert r.returncode == 0, r.stderr[-2000:]
        got.append(np.load(path))
    a, b = got
    assert sorted(a.files) == sorted(b.files)
    for name in a.files:
        if name.startswith("rain"):
            np.testing.assert_allclose(a[name], b[name], rtol=2.0**-22)
        else:
            assert np.array_equal(a[name], b[name]), name
