"""Timed cases of the solver: the calls that programs built on this package make, over their range of sizes.

Each case is one public call (or the calls of one loop iteration) with fresh
outputs, on inputs made from a seed with plain torch:

* the functional API on a small grid (``compute_cfl_dt`` + ``finite_volume_step``);
* whole forecasts (``run``, ``run_to_host``) and blocks of CFL-limited steps
  (``advance``) in exact arithmetic, the solver's default, and in fast arithmetic;
* a batched ensemble of members of uneven size (``B200Ensemble.advance_``);
* gradients: the gauge rollout and the physics interval of the trained coupling;
* the coupling around the physics: features, correction, output fields, and a
  whole physics + corrector interval of an ensemble.

``exact`` restates the scheme in float64 torch (the operation order of
``src/hybrid_flood/numpy_solver/shallow_water_2d.py:66-327``).
"""

from __future__ import annotations

import math
import os
import sys

import numpy as np
import torch

MM_HR = 1.0e-3 / 3600.0
DEV = "cuda"


# ---------------------------------------------------------------------------
# Cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # One iteration of a caller's own time loop on a small catchment grid
        # (irregular domain mask): latency and launches count.
        dict(name="step_96x130_exact", kind="step", terrain="catchment", rows=96, cols=130, arith="exact"),
        # The plain forecast configuration: 256^2 tilted plane with bumps under steady
        # rain, an output every 100 s, default (exact) arithmetic.  It starts ponded:
        # from a dry start the film stays millimetres deep, and its momenta follow
        # the rounding of depth + bed, so that two correct runs differ by parts in 10^4.
        dict(name="run_256_exact", kind="run", terrain="bumps", rows=256, cols=256, arith="exact", seconds=300.0,
             outputs=4),
        # A forecast on the reference's production grid size (517 x 551, masked, dx = 10 m).
        dict(name="run_517x551_exact", kind="run", terrain="catchment", rows=517, cols=551, arith="exact",
             seconds=300.0, outputs=4),
        # Steps of the urban scenario at scale in the solver's default arithmetic.
        dict(name="advance_2048_exact", kind="advance", terrain="urban", rows=2048, cols=2048, arith="exact", steps=32),
        # A block of steps on an ordinary ragged grid in fast arithmetic.
        dict(name="advance_300x420_fast", kind="advance", terrain="urban", rows=300, cols=420, arith="fast", steps=100),
        # The urban scenario at scale in fast arithmetic, from device to device.
        dict(name="advance_2048_fast", kind="advance", terrain="urban", rows=2048, cols=2048, arith="fast", steps=200),
        # The same as a forecast from and to pinned host memory (two outputs after the start).
        dict(name="host_2048_fast", kind="host", terrain="urban", rows=2048, cols=2048, arith="fast", seconds=60.0,
             outputs=3),
        # A batch of rainfall/roughness scenarios: 24 urban members of the four ensemble shapes.
        dict(name="ensemble_24_fast", kind="ensemble", members=24, scale=1.0, arith="fast", steps=50),
        # Calibration: gauge depths of a 512^2 fixed-dt rollout and their gradients
        # for Manning n, the initial depth and the rain scale.
        dict(name="gauge_512_exact", kind="gauge", rows=512, cols=512, arith="exact", steps=100),
        # The solver block of one training interval, forward and backward.
        dict(name="interval_512_fast", kind="interval", terrain="urban", rows=512, cols=512, arith="fast", seconds=6.0),
        # The passes around the physics of one coupled interval on a large grid:
        # features, three-channel correction and the output fields.
        dict(name="coupling_2048", kind="coupling", terrain="urban", rows=2048, cols=2048, arith="exact",
             layout="reference6", bf16=False, channels=3),
        # A coupled ensemble forecast: features, physics, bf16 corrector, correction, two intervals.
        dict(name="hybrid_4x512_fast", kind="hybrid", members=4, rows=512, cols=512, arith="fast", seconds=20.0),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step", "run", "advance", "advance", "host", "ensemble", "gauge", "interval", "coupling",
                       "hybrid"])
    arith = rng.choice(["exact", "fast"])
    if kind == "step":
        return dict(kind=kind, terrain=rng.choice(["catchment", "urban"]), rows=_log_int(rng, 24, 700),
                    cols=_log_int(rng, 24, 700), arith=arith)
    if kind == "run":
        return dict(kind=kind, terrain=rng.choice(["bumps", "catchment"]), rows=_log_int(rng, 96, 640),
                    cols=_log_int(rng, 96, 640), arith=arith, seconds=float(rng.randint(100, 300)),
                    outputs=rng.randint(2, 6))
    if kind == "advance":
        return dict(kind=kind, terrain="urban", rows=_log_int(rng, 128, 2048), cols=_log_int(rng, 128, 2048),
                    arith=arith, steps=rng.randint(16, 32) if arith == "exact" else rng.randint(32, 150))
    if kind == "host":
        return dict(kind=kind, terrain="urban", rows=_log_int(rng, 256, 2048), cols=_log_int(rng, 256, 2048),
                    arith="fast", seconds=float(rng.randint(10, 50)), outputs=rng.randint(2, 3))
    if kind == "ensemble":
        return dict(kind=kind, members=rng.randint(3, 20), scale=rng.choice([0.25, 0.5, 1.0]), arith="fast",
                    steps=rng.randint(20, 50))
    if kind == "gauge":
        return dict(kind=kind, rows=_log_int(rng, 96, 512), cols=_log_int(rng, 96, 512), arith="exact",
                    steps=10 * rng.randint(3, 10))
    if kind == "interval":
        return dict(kind=kind, terrain="urban", rows=_log_int(rng, 96, 512), cols=_log_int(rng, 96, 512), arith="fast",
                    seconds=float(rng.randint(3, 6)))
    if kind == "coupling":
        layout = rng.choice(["reference6", "state5"])
        return dict(kind=kind, terrain=rng.choice(["urban", "catchment"]), rows=_log_int(rng, 128, 2048),
                    cols=_log_int(rng, 128, 2048), arith="exact", layout=layout, bf16=rng.random() < 0.5,
                    channels=3 if layout == "reference6" else 1)
    return dict(kind=kind, members=rng.randint(1, 4), rows=8 * rng.randint(12, 64), cols=8 * rng.randint(12, 64),
                arith="fast", seconds=float(rng.randint(8, 20)))


# ---------------------------------------------------------------------------
# Inputs (plain torch and numpy, from the seed)
# ---------------------------------------------------------------------------
def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed) & 0x7FFFFFFFFFFF)
    return g


def _smooth(g, rows, cols, cell=24):
    """A smooth random field in about [-1, 1] (bilinear noise of `cell`-cell wavelength)."""
    r, c = max(2, rows // cell + 2), max(2, cols // cell + 2)
    n = torch.rand((1, 1, r, c), generator=g, device=DEV, dtype=torch.float64) * 2.0 - 1.0
    return torch.nn.functional.interpolate(n, size=(rows, cols), mode="bilinear", align_corners=True)[0, 0]


def _blocks(g, rows, cols):
    """Rectangles of 5 to 20 cells a side on about 30 % of the cells."""
    k = max(1, int(0.357 * rows * cols / 156.25))
    side = torch.randint(5, 21, (2, k), generator=g, device=DEV)
    h, w = side[0].clamp(max=rows), side[1].clamp(max=cols)
    r0 = (torch.rand(k, generator=g, device=DEV, dtype=torch.float64) * (rows - h + 1)).long()
    c0 = (torch.rand(k, generator=g, device=DEV, dtype=torch.float64) * (cols - w + 1)).long()
    d = torch.zeros((rows + 1, cols + 1), dtype=torch.int32, device=DEV)
    one = torch.ones(k, dtype=torch.int32, device=DEV)
    for r, c, s in ((r0, c0, one), (r0 + h, c0, -one), (r0, c0 + w, -one), (r0 + h, c0 + w, one)):
        d.index_put_((r, c), s, accumulate=True)
    return d.cumsum(0).cumsum(1)[:rows, :cols] > 0


def _fields(terrain, rows, cols, seed):
    """Bed, roughness, mask, state and controls of one domain, float32 on the device."""
    g = _gen(seed)
    rng = np.random.default_rng(seed)
    x = (torch.arange(cols, dtype=torch.float64, device=DEV) + 0.5)[None, :]
    y = (torch.arange(rows, dtype=torch.float64, device=DEV) + 0.5)[:, None]
    ones = torch.ones((rows, cols), dtype=torch.bool, device=DEV)
    times = np.arange(181, dtype=np.float64) * 60.0
    rates = rng.gamma(0.8, 6.0, 181) * MM_HR
    ctl = dict(gravity_m_s2=9.81, cfl=0.9, dry_tolerance_m=1.0e-3, max_dt_s=10.0, default_rainfall_m_s=0.0,
               boundary=(0, 1, 0, 0))
    if terrain == "bumps":  # tilted plane and 8 bumps, ponded, steady rain
        dx = 2.0
        bed = 0.005 * (cols * dx - x * dx) * torch.ones_like(y)
        for _ in range(8):
            a, s = rng.uniform(-0.5, 0.5), rng.uniform(10.0, 30.0)
            cx, cy = rng.uniform(0, cols * dx), rng.uniform(0, rows * dx)
            bed = bed + a * torch.exp(-((x * dx - cx) ** 2 + (y * dx - cy) ** 2) / (2 * s * s))
        man = torch.full_like(bed, 0.03)
        mask = ones
        depth = 0.15 + 0.05 * _smooth(g, rows, cols)
        u = v = torch.zeros_like(bed)
        times, rates = np.array([0.0, 600.0]), np.array([20.0, 20.0]) * MM_HR
    elif terrain == "urban":  # streets between raised blocks, ponded and flowing
        dx = 1.0
        blocks = _blocks(g, rows, cols)
        bed = 0.003 * (cols * dx - x * dx) + torch.where(blocks, 10.0, -0.2)
        man = torch.where(blocks, 0.05, 0.015).double()
        mask = ones
        depth = torch.where(blocks, 0.0, 0.12 + 0.08 * _smooth(g, rows, cols))
        u, v = 0.3 * _smooth(g, rows, cols), 0.3 * _smooth(g, rows, cols)
    else:  # catchment: irregular mask, valleys, dx = 10 m
        dx = 10.0
        bed = 0.002 * (cols * dx - x * dx) + 1.5 * _smooth(g, rows, cols, 60)
        man = 0.035 * torch.exp(0.3 * _smooth(g, rows, cols, 12))
        rr = ((x - cols / 2) / (0.49 * cols)) ** 2 + ((y - rows / 2) / (0.49 * rows)) ** 2
        mask = rr + 0.12 * _smooth(g, rows, cols, 30) < 1.0
        depth = torch.clamp_min(0.6 * _smooth(g, rows, cols, 40) + 0.1, 0.0)
        u, v = 0.2 * _smooth(g, rows, cols), 0.2 * _smooth(g, rows, cols)
        ctl.update(cfl=0.45, dry_tolerance_m=1.0e-4, boundary=(0, 1, 1, 0))
    f32 = lambda t: t.to(torch.float32).contiguous()  # noqa: E731
    h = f32(torch.where(mask, depth, torch.zeros_like(depth)))
    return dict(bed=f32(bed), manning_n=f32(man), domain_mask=mask, resolution_m=dx,
                rainfall_times_s=times.astype(np.float32), rainfall_rates_m_s=rates.astype(np.float32), **ctl), (
        h, f32(h * u.float()), f32(h * v.float()))


def _package():
    path = os.path.join(os.getcwd(), "gpu-hybrid-flood-forecasting_b200")
    if path not in sys.path:
        sys.path.insert(1, path)


ENSEMBLE_SHAPES = ((256, 256), (512, 512), (1024, 1024), (768, 1536))


def _shapes(case):
    if case["kind"] == "hybrid":
        return [(case["rows"], case["cols"])] * case["members"]
    return [tuple(int(s * case["scale"]) for s in ENSEMBLE_SHAPES[m % 4]) for m in range(case["members"])]


def _gauge_inputs(case, seed):
    kw, _ = _fields("bumps", case["rows"], case["cols"], seed)
    g = _gen(seed + 17)
    rows, cols = case["rows"], case["cols"]
    n = (0.03 * torch.exp(0.3 * _smooth(g, rows, cols, 9))).float()
    h0 = torch.clamp_min(1.0 - kw["bed"], 0.2) + 0.02 * _smooth(g, rows, cols).float()
    hu0 = h0 * (0.1 + 0.05 * _smooth(g, rows, cols).float())
    hv0 = h0 * (0.05 * _smooth(g, rows, cols).float() - 0.1)
    idx = torch.randperm(rows * cols, generator=g, device=DEV)[:16]
    w = torch.rand((case["steps"] // 10, 16), generator=g, device=DEV, dtype=torch.float32) - 0.5
    kw["manning_n"] = n
    return kw, n, h0.contiguous(), hu0.contiguous(), hv0.contiguous(), idx, w


def _cotangents(case, seed):
    g = _gen(seed + 29)
    return [_smooth(g, case["rows"], case["cols"], 8).float() for _ in range(3)]


def _coupling_inputs(case, seed):
    g = _gen(seed + 41)
    rows, cols, nch = case["rows"], case["cols"], case["channels"]
    res = torch.randn((rows, cols, nch), generator=g, device=DEV) * 0.02
    res = res.to(torch.bfloat16 if case["bf16"] else torch.float32)
    terrain, rough = _smooth(g, rows, cols).float(), _smooth(g, rows, cols).float()
    n = 3 if case["layout"] == "reference6" else 5
    mean = np.array([0.1, 0.01, -0.01, 3.0, 5.0], np.float32)[:n]
    std = np.array([0.08, 0.2, 0.15, 4.0, 5.0], np.float32)[:n]
    return res, terrain, rough, mean, std


WIDTHS = (32, 64, 128, 256)


def _net_weights(seed):
    """Weights of the 4-level corrector (5 -> 1 channels), rounded to bfloat16; submodule names of the package."""
    g = _gen(seed + 53)
    w = {}

    def conv(name, cout, cin, k, transposed=False, scale=1.0):
        shape = (cin, cout, k, k) if transposed else (cout, cin, k, k)
        fan = cin if transposed else cin * k * k
        w[name + ".weight"] = (torch.randn(shape, generator=g, device=DEV) * scale * (1.6 / fan) ** 0.5).bfloat16()
        w[name + ".bias"] = (torch.randn(cout, generator=g, device=DEV) * 0.05 * scale).bfloat16()

    cin = 5
    for lv, c in enumerate(WIDTHS):
        conv(f"encoders.{lv}.conv_1", c, cin, 3)
        conv(f"encoders.{lv}.conv_2", c, c, 3)
        if lv < 3:
            conv(f"downsample.{lv}", WIDTHS[lv + 1], c, 2)
            cin = WIDTHS[lv + 1]
    cin = WIDTHS[-1]
    for i, c in enumerate(reversed(WIDTHS[:-1])):
        conv(f"upsample.{i}", c, cin, 2, transposed=True)
        conv(f"decoders.{i}.conv_1", c, 2 * c, 3)
        conv(f"decoders.{i}.conv_2", c, c, 3)
        cin = c
    conv("residual_head", 1, cin, 1, scale=0.01)
    return w


HYBRID_STATS = (np.array([0.1, 0.0, 0.0, 3.0, 5.0], np.float32), np.array([0.1, 0.05, 0.05, 5.0, 5.0], np.float32),
                np.array([0.01], np.float32))


# ---------------------------------------------------------------------------
# State, pass, work
# ---------------------------------------------------------------------------
def prepare(case, seed):
    _package()
    from hybrid_flood_b200.ensemble import B200Ensemble
    from hybrid_flood_b200.hybrid import HybridInputs
    from hybrid_flood_b200.solver import B200ShallowWaterSolver, SWEState

    kind = case["kind"]
    s = dict(case=dict(case))
    if kind in ("ensemble", "hybrid"):
        made = [_fields("urban", r, c, 1000 * seed + m) for m, (r, c) in enumerate(_shapes(case))]
        s["ens"] = B200Ensemble([kw for kw, _ in made], arithmetic=case["arith"])
        s["states"] = [SWEState(*st) for _, st in made]
        if kind == "hybrid":
            from hybrid_flood_b200.unet import corrector_4level

            net = corrector_4level()
            net.load_state_dict(_net_weights(seed))
            s["net"] = net.to(device=DEV, dtype=torch.bfloat16, memory_format=torch.channels_last).eval()
            s["inputs"] = HybridInputs(None, None, HYBRID_STATS[0], HYBRID_STATS[1], 25.0, HYBRID_STATS[2])
        return s
    if kind == "gauge":
        kw, n, h0, hu0, hv0, idx, w = _gauge_inputs(case, seed)
        s.update(n=n.requires_grad_(True), h0=h0.requires_grad_(True), hu0=hu0, hv0=hv0, idx=idx, w=w,
                 scale=torch.tensor(1.0, device=DEV, requires_grad=True))
    else:
        kw, st = _fields(case["terrain"], case["rows"], case["cols"], seed)
        s["state"] = SWEState(*st)
    kw = {k: v.detach() if isinstance(v, torch.Tensor) else v for k, v in kw.items()}
    s["solver"] = B200ShallowWaterSolver(kw.pop("bed"), kw.pop("manning_n"), kw.pop("domain_mask"), **kw,
                                         arithmetic=case["arith"])
    if kind in ("run", "host"):
        s["times"] = np.linspace(0.0, case["seconds"], case["outputs"]).astype(np.float32)
    if kind == "host":
        s["host"] = tuple(t.cpu().pin_memory() for t in s["state"])
        s["out"] = [torch.empty((case["outputs"], case["rows"], case["cols"])).pin_memory() for _ in range(3)]
    if kind == "interval":
        s["cot"] = _cotangents(case, seed)
        s["leaves"] = [t.clone().requires_grad_(True) for t in s["state"]]
    if kind == "coupling":
        res, terrain, rough, mean, std = _coupling_inputs(case, seed)
        s["residual"] = res
        planes = (terrain, rough) if case["layout"] == "reference6" else (None, None)
        s["inputs"] = HybridInputs(*planes, mean, std, 25.0, None)
    return s


def run(s):
    from hybrid_flood_b200 import adjoint, hybrid, output, solver, training

    case = s["case"]
    kind = case["kind"]
    if kind == "step":
        dt = solver.compute_cfl_dt(s["state"], s["solver"].params)
        return tuple(solver.finite_volume_step(s["state"], s["solver"].params, dt, 90.0)), dt
    if kind == "run":
        return tuple(s["solver"].run(s["state"], s["times"]).states)
    if kind == "host":
        return tuple(s["solver"].run_to_host(s["host"], s["times"], out=s["out"]).states)
    if kind == "advance":
        return tuple(s["solver"].advance(s["state"], case["steps"], 1800.0)[0])
    if kind == "ensemble":
        cur = [solver.SWEState(*(t.clone() for t in st)) for st in s["states"]]
        s["ens"].advance_(cur, case["steps"], [1800.0] * len(cur))
        # All members' cells of a quantity in one array.
        return [torch.cat([st[q].reshape(-1) for st in cur]) for q in range(3)]
    if kind == "gauge":
        obs = adjoint.gauge_rollout(s["solver"], s["n"], s["h0"], s["scale"], hu0=s["hu0"], hv0=s["hv0"],
                                    n_steps=case["steps"], dt=0.2, gauge_index=s["idx"], obs_every=10,
                                    checkpoint_every=50)
        grads = torch.autograd.grad(obs, (s["n"], s["h0"], s["scale"]), s["w"])
        return obs.detach(), grads
    if kind == "interval":
        st, _ = training.physics_interval(s["solver"], s["leaves"], 1800.0, 1800.0 + case["seconds"], 2000)
        grads = torch.autograd.grad(tuple(st), s["leaves"], s["cot"])
        return [t.detach() for t in st], grads
    if kind == "coupling":
        f = hybrid.network_features(s["solver"], s["state"], s["inputs"], 1800.0, layout=case["layout"],
                                    dtype=torch.bfloat16 if case["bf16"] else torch.float32)
        c = hybrid.apply_residual_correction(s["solver"], s["state"], s["residual"], correction_relaxation=0.3,
                                             clip_limits=[0.05] * case["channels"])
        return f, tuple(c), output.output_fields(s["solver"], c)
    times = np.array([0.0, case["seconds"], 2.0 * case["seconds"]])
    traj, _ = hybrid.run_coupled_ensemble(s["ens"], s["states"], s["net"], s["inputs"], times,
                                          max_substeps_per_interval=2000, correction_relaxation=0.5, keep_states=False)
    return [torch.stack([tr[q] for tr in traj]) for q in range(3)]


#: Bytes of a forward step per cell (h, hu, hv, bed, n^2 in; h, hu, hv out) and
#: about how many operations it takes (five faces' worth of flux arithmetic and the update).
STEP_BYTES, STEP_FLOPS = 32.0, 260.0
#: Steps a second of simulated time takes on the terrains (dt of the CFL condition at their depths).
STEPS_PER_S = {"bumps": 2.4, "urban": 4.2, "catchment": 1.5}
NET_FLOPS_PER_CELL = 2.0 * 9 * (5 * 32 + 32 * 32 + 64 * 32 + 32 * 32
                                + (64 * 64 * 2 + 128 * 64 + 64 * 64) / 4
                                + (128 * 128 * 2 + 256 * 128 + 128 * 128) / 16 + (256 * 256 * 2) / 64)


def work(case):
    kind = case["kind"]
    if kind in ("ensemble", "hybrid"):
        cells = float(sum(r * c for r, c in _shapes(case)))
    else:
        cells = float(case["rows"] * case["cols"])
    if kind == "step":
        return {"bytes": cells * (STEP_BYTES + 16.0), "flops": cells * (STEP_FLOPS + 12.0)}
    if kind == "coupling":
        es = 2.0 if case["bf16"] else 4.0
        nf = 6 if case["layout"] == "reference6" else 5
        feats = 12.0 + 4.0 + (8.0 if nf == 6 else 4.0) + nf * es
        return {"bytes": cells * (feats + (16.0 + es * case["channels"] + 12.0) + 32.0), "flops": cells * 60.0}
    if kind in ("advance", "ensemble"):
        steps = case["steps"]
    elif kind == "gauge":  # forward, recomputation, reverse
        return {"bytes": cells * case["steps"] * (2 * STEP_BYTES + 52.0), "flops": cells * case["steps"] * 4 * STEP_FLOPS}
    else:
        terrain = case.get("terrain", "urban")
        steps = case["seconds"] * STEPS_PER_S[terrain] * (2.0 if kind == "hybrid" else 1.0)
    if kind == "interval":
        return {"bytes": cells * steps * (2 * STEP_BYTES + 52.0), "flops": cells * steps * 4 * STEP_FLOPS}
    w = {"bytes": cells * steps * STEP_BYTES, "flops": cells * steps * STEP_FLOPS}
    if kind == "hybrid":
        w["flops"] += 2.0 * cells * NET_FLOPS_PER_CELL
        w["bytes"] += 2.0 * cells * 100.0
    if kind == "host":
        w["bytes"] += cells * 12.0 * (1 + case["outputs"])
    return w


# ---------------------------------------------------------------------------
# Float64 restatement
# ---------------------------------------------------------------------------
class _Domain64:
    def __init__(self, kw):
        d = lambda t: t.detach().to(DEV, torch.float64)  # noqa: E731
        f = lambda x: float(np.float32(x))  # noqa: E731
        self.z, self.n2 = d(kw["bed"]), d(kw["manning_n"]) ** 2
        self.mask = kw["domain_mask"].to(DEV)
        self.dx = kw["resolution_m"]
        self.g, self.dry, self.cfl, self.max_dt = kw["gravity_m_s2"], f(kw["dry_tolerance_m"]), kw["cfl"], kw["max_dt_s"]
        self.bnd = kw["boundary"]
        self.rt, self.rr = kw["rainfall_times_s"].astype(np.float64), kw["rainfall_rates_m_s"].astype(np.float64)
        self.default = kw["default_rainfall_m_s"]
        pad = lambda t: torch.nn.functional.pad(t[None, None].double(), (1, 1, 1, 1), mode="replicate")[0, 0]  # noqa: E731
        self.zg, self.mg = pad(self.z), pad(self.mask) > 0.5

    def rain(self, t):
        return float(np.interp(t, self.rt, self.rr, left=self.default, right=self.default))


def _root(x):
    """sqrt with a zero derivative at zero."""
    pos = x > 0
    return torch.where(pos, torch.sqrt(torch.where(pos, x, torch.ones_like(x))), torch.zeros_like(x))


def _over(m, h, wet):
    return torch.where(wet, m / torch.where(wet, h, torch.ones_like(h)), torch.zeros_like(m))


def _face64(D, lo, hi, axis):
    """HLL flux of every face between lo and hi cells, and the pressure corrections of both sides."""
    (hL, uL, vL, zL, aL), (hR, uR, vR, zR, aR) = lo, hi
    hw, lw = aL & ~aR, ~aL & aR
    su, sv = (-1.0, 1.0) if axis == 1 else (1.0, -1.0)
    hL, hR = torch.where(lw, hR, hL), torch.where(hw, hL, hR)
    zL, zR = torch.where(lw, zR, zL), torch.where(hw, zL, zR)
    uL, uR = torch.where(lw, su * uR, uL), torch.where(hw, su * uL, uR)
    vL, vR = torch.where(lw, sv * vR, vL), torch.where(hw, sv * vL, vR)
    zf = torch.maximum(zL, zR)
    HL, HR = torch.relu(hL + zL - zf), torch.relu(hR + zR - zf)
    XL, YL, XR, YR = HL * uL, HL * vL, HR * uR, HR * vR
    zero = torch.zeros_like(HL)
    wL, wR = HL > D.dry, HR > D.dry
    uL, vL, uR, vR = (torch.where(w, a, zero) for w, a in ((wL, uL), (wL, vL), (wR, uR), (wR, vR)))
    nL, nR = (uL, uR) if axis == 1 else (vL, vR)
    cL, cR = _root(D.g * HL), _root(D.g * HR)
    sL, sR = torch.minimum(nL - cL, nR - cR), torch.maximum(nL + cL, nR + cR)
    pL, pR = 0.5 * D.g * HL * HL, 0.5 * D.g * HR * HR
    if axis == 1:
        fL, fR = (XL, XL * nL + pL, XL * vL), (XR, XR * nR + pR, XR * vR)
    else:
        fL, fR = (YL, XL * nL, YL * nL + pL), (YR, XR * nR, YR * nR + pR)
    den = torch.where(sR - sL > 1.0e-12, sR - sL, torch.ones_like(sL))
    rel = aL | aR
    out = []
    for a, b, p, q in zip(fL, fR, (HL, XL, YL), (HR, XR, YR)):
        m = (sR * a - sL * b + sL * sR * (q - p)) / den
        out.append(torch.where(rel, torch.where(sL >= 0, a, torch.where(sR <= 0, b, m)), zero))
    cl = torch.where(rel, 0.5 * D.g * (hL * hL - HL * HL), zero)
    cr = torch.where(rel, 0.5 * D.g * (hR * hR - HR * HR), zero)
    return out, cl, cr


def _step64(D, st, dt, t, n2=None, rain_scale=1.0):
    h, hu, hv = st
    n2 = D.n2 if n2 is None else n2
    pad = lambda a: torch.nn.functional.pad(a[None, None], (1, 1, 1, 1), mode="replicate")[0, 0]  # noqa: E731
    H, U, V = pad(h), pad(hu), pad(hv)
    sx, sy = torch.ones_like(H), torch.ones_like(H)
    for k, (s, sl) in enumerate(((sx, (slice(None), 0)), (sx, (slice(None), -1)), (sy, (0, slice(None))),
                                 (sy, (-1, slice(None))))):
        if D.bnd[k] == 0:
            s[sl] = -1.0
    U, V = U * sx, V * sy
    wet = H > D.dry
    cell = (H, _over(U, H, wet), _over(V, H, wet), D.zg, D.mg)
    at = lambda r, c: tuple(a[r, c] for a in cell)  # noqa: E731
    inner = slice(1, -1)
    fx, cxl, cxr = _face64(D, at(inner, slice(None, -1)), at(inner, slice(1, None)), 1)
    fy, cyl, cyr = _face64(D, at(slice(None, -1), inner), at(slice(1, None), inner), 0)
    upd = []
    for q, a in enumerate((h, hu, hv)):
        right, left = fx[q][:, 1:], fx[q][:, :-1]
        top, bot = fy[q][1:], fy[q][:-1]
        if q == 1:
            right, left = right + cxl[:, 1:], left + cxr[:, :-1]
        if q == 2:
            top, bot = top + cyl[1:], bot + cyr[:-1]
        upd.append(a - dt * ((right - left) / D.dx + (top - bot) / D.dx))
    zero = torch.zeros_like(h)
    u0 = upd[0] + torch.where(D.mask, dt * D.rain(t) * rain_scale * torch.ones_like(h), zero)
    hn = torch.relu(u0)
    norm = _root(upd[1] ** 2 + upd[2] ** 2)
    deep = torch.where(hn > D.dry, hn, torch.full_like(hn, D.dry))
    den = 1.0 + dt * D.g * n2 * norm / deep ** float(np.float32(7.0 / 3.0))
    keep = D.mask & (hn > D.dry)
    return (torch.where(D.mask, hn, zero), torch.where(keep, upd[1] / den, zero),
            torch.where(keep, upd[2] / den, zero))


def _cfl64(D, st):
    h, hu, hv = (a.detach() for a in st)
    wet = h > D.dry
    w = torch.sqrt(D.g * h.clamp_min(0.0))
    inv = (_over(hu, h, wet).abs() + w) / D.dx + (_over(hv, h, wet).abs() + w) / D.dx
    m = float(torch.where(D.mask, inv, torch.zeros_like(inv)).max())
    return min(D.cfl / m, D.max_dt) if m > 0 else D.max_dt


def _advance64(D, st, t, target=None, steps=None):
    k = 0
    while (target is not None and t < target - 1.0e-7) or (steps is not None and k < steps):
        dt = _cfl64(D, st)
        if target is not None:
            dt = min(dt, target - t)
        st = _step64(D, st, dt, t)
        t += dt
        k += 1
    return st


def _double(st):
    return tuple(t.detach().to(DEV, torch.float64) for t in st)


def _features64(D, st, layout, mean, std, rain, terrain, rough):
    """Features in float64 (the rain channel as the float32 value the path feeds the network)."""
    h, hu, hv = st
    m, s = (torch.from_numpy(a.astype(np.float64)).to(DEV) for a in (mean, std))
    zero = torch.zeros_like(h)
    if layout == "reference6":
        wet = h > D.dry
        ch = [h, _over(hu, h, wet), _over(hv, h, wet)]
        ch = [torch.where(D.mask, (a - m[q]) / s[q], zero) for q, a in enumerate(ch)]
        return torch.stack(ch + [torch.full_like(h, rain / 25.0), terrain.double(), rough.double()], -1)
    src = [h, hu, hv, D.z, torch.full_like(h, rain)]
    return torch.stack([torch.where(D.mask, (a - m[q]) / s[q], zero) for q, a in enumerate(src)], -1)


def _correct64(D, st, res, relax, lim):
    h, hu, hv = st
    zero = torch.zeros_like(h)
    r = [res[..., q].double().clamp(-lim[q], lim[q]) for q in range(res.shape[-1])]
    wet = h > D.dry
    u, v = _over(hu, h, wet), _over(hv, h, wet)
    prov = torch.where(D.mask, torch.relu(h + relax * r[0]), zero)
    target, have = torch.where(D.mask, h, zero).sum(), prov.sum()
    eps = float(np.finfo(np.float32).eps)
    ch = prov * (target / have if have > eps else 1.0) if target > eps else h
    if len(r) == 3:
        u, v = u + relax * r[1], v + relax * r[2]
    keep = D.mask & (ch > D.dry)
    return ch, torch.where(keep, ch * u, zero), torch.where(keep, ch * v, zero)


def _net64(w, x):
    F = torch.nn.functional
    p = {k: v.double() for k, v in w.items()}
    conv = lambda x, name, **kw: F.conv2d(x, p[name + ".weight"], p[name + ".bias"], **kw)  # noqa: E731

    def pair(x, name):
        return torch.relu(conv(torch.relu(conv(x, name + ".conv_1", padding=1)), name + ".conv_2", padding=1))

    skips = []
    for lv in range(4):
        x = pair(x, f"encoders.{lv}")
        skips.append(x)
        if lv < 3:
            x = conv(F.pad(x, (0, x.shape[-1] % 2, 0, x.shape[-2] % 2)), f"downsample.{lv}", stride=2)
    for i in range(3):
        skip = skips[2 - i]
        x = F.conv_transpose2d(x, p[f"upsample.{i}.weight"], p[f"upsample.{i}.bias"], stride=2)
        if x.shape[-2:] != skip.shape[-2:]:
            x = F.interpolate(x, size=skip.shape[-2:], mode="bilinear", align_corners=False)
        x = pair(torch.cat((x, skip), 1), f"decoders.{i}")
    return conv(x, "residual_head")


def exact(case, seed):
    kind = case["kind"]
    if kind == "gauge":
        kw, n, h0, hu0, hv0, idx, w = _gauge_inputs(case, seed)
        D = _Domain64(kw)
        nn, hh = n.double().requires_grad_(True), h0.double().requires_grad_(True)
        sc = torch.tensor(1.0, dtype=torch.float64, device=DEV, requires_grad=True)
        st, obs, t = (hh, hu0.double(), hv0.double()), [], 0.0
        for k in range(case["steps"]):
            st = _step64(D, st, 0.2, t, nn ** 2, sc)
            t += 0.2
            if (k + 1) % 10 == 0:
                obs.append(st[0].reshape(-1)[idx])
        obs = torch.stack(obs)
        grads = torch.autograd.grad(obs, (nn, hh, sc), w.double())
        return obs.detach(), grads
    with torch.no_grad():
        if kind == "ensemble":
            out = []
            for m, (r, c) in enumerate(_shapes(case)):
                kw, st = _fields("urban", r, c, 1000 * seed + m)
                out.append(_advance64(_Domain64(kw), _double(st), 1800.0, steps=case["steps"]))
            return [torch.cat([st[q].reshape(-1) for st in out]) for q in range(3)]
        if kind == "hybrid":
            w = _net_weights(seed)
            mean, std, rstd = HYBRID_STATS
            made = [_fields("urban", r, c, 1000 * seed + m) for m, (r, c) in enumerate(_shapes(case))]
            out = []
            for kw, st in made:
                D, st = _Domain64(kw), _double(st)
                for k in range(2):
                    t = k * case["seconds"]
                    f = _features64(D, st, "state5", mean, std, D.rain(t) * 3.6e6, None, None)
                    st = _advance64(D, st, t, target=t + case["seconds"])
                    r = _net64(w, f.permute(2, 0, 1)[None])[0].permute(1, 2, 0)
                    st = _correct64(D, st, r, 0.5, [5.0 * float(rstd[0])])
                out.append(st)
            return [torch.stack([st[q] for st in out]) for q in range(3)]
        kw, st32 = _fields(case["terrain"], case["rows"], case["cols"], seed)
        D, st = _Domain64(kw), _double(st32)
        if kind == "step":
            dt = _cfl64(D, st)
            return _step64(D, st, dt, 90.0), dt
        if kind == "advance":
            return _advance64(D, st, 1800.0, steps=case["steps"])
        if kind in ("run", "host"):
            times = np.linspace(0.0, case["seconds"], case["outputs"]).astype(np.float32).astype(np.float64)
            outs = [st]
            for a, b in zip(times[:-1], times[1:]):
                outs.append(_advance64(D, outs[-1], float(a), target=float(b)))
            return tuple(torch.stack([o[q] for o in outs]) for q in range(3))
        if kind == "coupling":
            res, terrain, rough, mean, std = _coupling_inputs(case, seed)
            f = _features64(D, st, case["layout"], mean, std, D.rain(1800.0) * 3.6e6, terrain, rough)
            lim = float(np.float32(0.05))
            c = _correct64(D, st, res, 0.3, [lim] * case["channels"])
            wet, nan = c[0] > D.dry, torch.full_like(c[0], float("nan"))
            u, v = _over(c[1], c[0], wet), _over(c[2], c[0], wet)
            m = lambda a: torch.where(D.mask, a, nan)  # noqa: E731
            return f[None], c, dict(depth=m(c[0]), x_velocity=m(u), y_velocity=m(v), velocity=m(torch.hypot(u, v)))
    # The interval's gradients: the steps' dt is held fixed in the reverse pass.
    leaves = [t.clone().requires_grad_(True) for t in st]
    end = _advance64(D, leaves, 1800.0, target=1800.0 + case["seconds"])
    grads = torch.autograd.grad(end, leaves, [c.double() for c in _cotangents(case, seed)])
    return [t.detach() for t in end], grads
