"""The work that users of this framework have it do, as timed cases.

``listed()`` names twelve of them, ``draw(rng)`` gives more of the same
ranges; ``prepare`` makes what a user's program holds before the call,
``run`` is one pass through the public entry points, ``work`` its least
bytes and operations and ``exact`` the same results in 64 bits by plain
torch.

Kinds of cases
  step       one ``SWE2D.step`` call, as a program with its own time loop
             makes it (any boundary type, friction law, batch, rainfall and
             infiltration; both arithmetic modes)
  forward    one ``SWE2D.forward`` call of some tens of CFL steps
  ensemble   ``Ensemble.run``: scenarios of uneven grids in one launch
  gauges     ``GaugeEnsemble.run``: the training runs of the warm start
  inversion  ``gauge_run`` forward and backward: one iteration of the
             boundary inversion (gauge misfit -> gradient of the levels), in
             the default arithmetic: a rounding moves the limiters' choices,
             and with them a gradient by up to 1e-3, so that gradients of
             the tolerance mode cannot be compared between two builds of it
  stepgrad   one ``SWE2D.step`` under autograd and its backward pass
  train      one ``WarmStartNet.train_step``
  predict    ``WarmStartNet.predict_controls`` of some gauge records
"""
from __future__ import annotations

import math

import torch

from diffswe2d_b200 import SWE2D, RainfallForcing, SWEConfig
from diffswe2d_b200 import scenarios
from diffswe2d_b200.ensemble import Ensemble, GaugeEnsemble
from diffswe2d_b200.gauge_run import gauge_run
from diffswe2d_b200.warmstart import (CONTROL_MEAN, CONTROL_SCALE, CONTROLS, GAUGES, INPUT_SCALE, SAMPLES,
                                      Conv, WarmStartNet, normalise_controls)

DEV = "cuda"

# Sides of the domain: the runup basin (inflow from the west), a closed
# basin, and an open catchment.
SIDES = {
    "runup": ("water_level", "wall", "wall", "wall"),
    "walls": ("wall", "wall", "wall", "wall"),
    "open": ("absorbing", "transmissive", "absorbing", "water_level"),
    "channel": ("periodic", "periodic", "wall", "wall"),
}
FLOPS_PER_STAGE = 320     # per cell: five limited increments and a flux per direction, the update
DX = 0.014                # spacing of the runup basin [m]
STEP_S = 0.0026           # about one CFL step of it [s]


def listed():
    return [
        # The smallest call: a patch of the runup basin stepped from a user's own loop.
        dict(name="step_64x96", kind="step", ny=64, nx=96, batch=1, arithmetic="exact", sides="runup",
             friction="manning", rain=False),
        # Rain on a catchment: rain and infiltration fields, roughness-length friction, open sides, odd sizes.
        dict(name="step_rain_2x611x517", kind="step", ny=611, nx=517, batch=2, arithmetic="exact",
             sides="open", friction="roughness_length", rain=True),
        # The runup basin advanced between two outputs.
        dict(name="forward_runup_244x393", kind="forward", ny=244, nx=393, dx=DX, arithmetic="fast",
             sides="runup", t_end=0.13, tiled=False),
        # A closed basin of a million cells in the default arithmetic, ragged sizes.
        dict(name="forward_walls_1021x1019", kind="forward", ny=1021, nx=1019, dx=DX, arithmetic="exact",
             sides="walls", t_end=0.042, tiled=False),
        # The benchmark's 4096 x 4096 grid.
        dict(name="forward_runup_4096x4096", kind="forward", ny=4096, nx=4096, dx=DX, arithmetic="fast",
             sides="runup", t_end=0.03, tiled=True),
        # A hazard ensemble: grids of uneven sides in one launch.
        dict(name="ensemble_24_fast", kind="ensemble", count=24, lo=128, hi=1024, sizes_seed=0, steps=40,
             arithmetic="fast"),
        # Training runs of the warm start.
        dict(name="gauges_64x122x196", kind="gauges", count=64, ny=122, nx=196, dx=2 * DX, n_out=8,
             arithmetic="fast"),
        # One iteration of the four-case inversion on the runup basin's grid.
        dict(name="inversion_4x244x393", kind="inversion", batch=4, ny=244, nx=393, dx=DX, n_out=14,
             arithmetic="exact", every=32, store=True),
        # The same at half the resolution, its segments recomputed instead of stored.
        dict(name="inversion_8x122x196", kind="inversion", batch=8, ny=122, nx=196, dx=2 * DX, n_out=14,
             arithmetic="exact", every=32, store=False),
        # A step differentiated by itself, as in a user's own differentiable loop.
        dict(name="stepgrad_2x244x393", kind="stepgrad", batch=2, ny=244, nx=393, arithmetic="exact",
             sides="runup"),
        # One training step of the warm start at its batch size.
        dict(name="train_256", kind="train", batch=256),
        # Warm starts of the hundred held-out cases.
        dict(name="predict_100", kind="predict", batch=100),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step", "forward", "forward", "ensemble", "gauges", "inversion", "stepgrad", "train",
                       "predict"])
    arithmetic = rng.choice(["exact", "fast"])
    if kind == "step":
        return dict(kind=kind, ny=_log(rng, 40, 1200), nx=_log(rng, 40, 1200), batch=rng.randint(1, 3),
                    arithmetic=arithmetic, sides=rng.choice(sorted(SIDES)),
                    friction=rng.choice(["manning", "roughness_length"]), rain=rng.random() < 0.3)
    if kind == "forward":
        ny, nx = _log(rng, 96, 3000), _log(rng, 96, 3000)
        steps = min(48, max(6, int(40e6 / (ny * nx))))
        return dict(kind=kind, ny=ny, nx=nx, dx=DX, arithmetic=arithmetic,
                    sides=rng.choice(["runup", "walls"]), t_end=round(steps * STEP_S, 5), tiled=False)
    if kind == "ensemble":
        return dict(kind=kind, count=rng.randint(8, 32), lo=128, hi=rng.choice([384, 512, 768]),
                    sizes_seed=rng.randint(1, 1 << 20), steps=rng.randint(20, 40), arithmetic=arithmetic)
    if kind == "gauges":
        ny, nx, dx = rng.choice([(61, 98, 4 * DX), (122, 196, 2 * DX)])
        return dict(kind=kind, count=_log(rng, 8, 128), ny=ny, nx=nx, dx=dx, n_out=rng.randint(4, 8),
                    arithmetic=arithmetic)
    if kind == "inversion":
        ny, nx, dx = rng.choice([(61, 98, 4 * DX), (122, 196, 2 * DX), (183, 295, 56 * DX / 42)])
        return dict(kind=kind, batch=rng.randint(1, 8), ny=ny, nx=nx, dx=dx, n_out=rng.randint(8, 14),
                    arithmetic="exact", every=32, store=rng.random() < 0.5)
    if kind == "stepgrad":
        return dict(kind=kind, batch=rng.randint(1, 4), ny=_log(rng, 48, 400), nx=_log(rng, 48, 400),
                    arithmetic="exact", sides=rng.choice(["runup", "walls"]))
    if kind == "train":
        return dict(kind=kind, batch=_log(rng, 32, 512))
    return dict(kind=kind, batch=_log(rng, 1, 700))


# ------------------------------------------------------------------ inputs
def _generator(seed):
    return torch.Generator().manual_seed(int(seed))


def _uniform(g, lo, hi, n):
    return (torch.rand(n, generator=g, dtype=torch.float64) * (hi - lo) + lo).tolist()


def _axes(ny, nx, dx):
    x = (torch.arange(nx, device=DEV, dtype=torch.float64) + 0.5) * dx
    y = (torch.arange(ny, device=DEV, dtype=torch.float64) + 0.5) * dx
    return x[None, :], y[:, None]


def _beach(g, ny, nx, dx, bumps=12):
    """A plane beach from 0.13 m below to 0.10 m above still water with Gaussian valleys and ridges."""
    x, y = _axes(ny, nx, dx)
    lx, ly = nx * dx, ny * dx
    z = (-0.13 + 0.23 * x / lx).expand(ny, nx).clone()
    cx, cy = _uniform(g, 0, lx, bumps), _uniform(g, 0, ly, bumps)
    amp, sig = _uniform(g, -0.03, 0.03, bumps), _uniform(g, 0.05, 0.15, bumps)
    for k in range(bumps):
        s = sig[k] * min(lx, ly)
        z += amp[k] * torch.exp(-(x - cx[k]) ** 2 / (2 * s * s)) * torch.exp(-(y - cy[k]) ** 2 / (2 * s * s))
    return z


def _waves(g, ny, nx, dx, amplitude, count=5):
    """A smooth field of a few waves some metres long."""
    x, y = _axes(ny, nx, dx)
    out = torch.zeros((ny, nx), device=DEV, dtype=torch.float64)
    kx, ky, ph = _uniform(g, 1, 5, count), _uniform(g, -4, 4, count), _uniform(g, 0, 6.28, count)
    for k in range(count):
        out += torch.sin(kx[k] * x + ky[k] * y + ph[k])
    return out * (amplitude / math.sqrt(count))


def _sea(g, z, dx):
    """[3, ny, nx] water in motion over the bed: waves of a centimetre, currents, wet and dry land."""
    ny, nx = z.shape
    h = torch.clamp(_waves(g, ny, nx, dx, 0.01) - z, min=0.0)
    u, v = _waves(g, ny, nx, dx, 0.12), _waves(g, ny, nx, dx, 0.08)
    return torch.stack([h, h * u, h * v])


def _site(g, batch, ny, nx, dx):
    """Beds [B,1,ny,nx] and states [B,3,ny,nx], float32."""
    beds = [_beach(g, ny, nx, dx) for _ in range(batch)]
    states = [_sea(g, z, dx) for z in beds]
    return (torch.stack(beds)[:, None].float().contiguous(), torch.stack(states).float().contiguous())


def _config(sides, friction="manning"):
    left, right, top, bottom = SIDES[sides]
    return SWEConfig(boundary_left=left, boundary_right=right, boundary_top=top, boundary_bottom=bottom,
                     frictionmodel=friction)


def _series(g):
    """A boundary series at 50 Hz (times, levels) of an N-wave with a seeded crest."""
    t = torch.arange(scenarios.RUNUP_SAMPLES, dtype=torch.float64) * scenarios.RUNUP_DT_SAMPLE
    crest = _uniform(g, 0.012, 0.018, 1)[0]
    w = crest * torch.sin(2 * math.pi * t / 15.0 + 0.3)
    return t.float().to(DEV), w.float().to(DEV)


def _model(bed, rough, dx, cfg, arithmetic, rainfall=None):
    return SWE2D(bed, rough, dx, dx, config=cfg, train_dem=False, arithmetic=arithmetic, rainfall=rainfall)


def _step_inputs(case, seed):
    g = _generator(seed)
    ny, nx, B = case["ny"], case["nx"], case["batch"]
    bed, _ = _site(g, 1, ny, nx, DX)  # one bed, several states of the water on it
    U = torch.stack([_sea(g, bed[0, 0].double(), DX) for _ in range(B)]).float().contiguous()
    rough = torch.full_like(bed, 0.01 if case["friction"] == "manning" else 0.002)
    rough *= 1 + 0.3 * _waves(g, ny, nx, DX, 1.0).float()
    rough.clamp_(min=1e-4)
    level = _uniform(g, -0.01, 0.01, 1)[0]
    rain = infil = None
    if case["rain"]:
        rates = torch.stack([_waves(g, ny, nx, DX, 1e-5) + 2e-5 for _ in range(3)]).clamp(min=0)
        rain = (torch.tensor([0.0, 60.0, 120.0], device=DEV), rates[:, None].float().contiguous())
        infil = (_waves(g, ny, nx, DX, 2e-6) + 3e-6).float()[None, None].contiguous()
    return bed, rough, U, level, rain, infil


def _forward_inputs(case, seed):
    g = _generator(seed)
    ny, nx, dx = case["ny"], case["nx"], case["dx"]
    if case["tiled"]:  # the stored state of the runup basin, tiled
        sc = scenarios.throughput_workload(ny, nx)
        bed, U = torch.from_numpy(sc.bed).to(DEV)[None, None], torch.from_numpy(sc.U0).to(DEV)
        U = U * (1 + 0.02 * _waves(g, ny, nx, dx, 1.0).float())
    else:
        bed, U = _site(g, 1, ny, nx, dx)
    return bed, torch.full_like(bed, 0.01), U.contiguous(), _series(g)


def _ensemble_inputs(case, seed):
    g = _generator(seed)
    out = []
    for ny, nx in scenarios.ensemble_sizes(case["count"], case["lo"], case["hi"], case["sizes_seed"]):
        dx = DX * 393 / nx
        z = _beach(g, ny, nx, dx)
        U = _sea(g, z, dx)
        inflow = _uniform(g, 0, 1, 1)[0] < 0.5
        times, levels = _series(g) if inflow else (None, None)
        n = _uniform(g, 0.01, 0.035, 1)[0]
        cfg = dict(zip(("boundary_left", "boundary_right", "boundary_top", "boundary_bottom"),
                       SIDES["runup" if inflow else "walls"]))
        out.append(scenarios.Scenario("member", z.float(), torch.full((ny, nx), n, device=DEV),
                                      U.float()[None], dx, dx, cfg, times, levels, case["steps"]))
    return out


def _gauge_cells(ny, nx):
    """Six gauges, the nearest a few cells off the inflow."""
    return [(int(ny * f), 2 + int(nx * e)) for f, e in
            ((0.2, 0.0), (0.5, 0.01), (0.8, 0.02), (0.35, 0.04), (0.65, 0.08), (0.5, 0.3))]


def _levels(g, batch, n_out):
    t = torch.arange(n_out, dtype=torch.float64) * scenarios.RUNUP_DT_SAMPLE
    rows = []
    for _ in range(batch):
        a, p = _uniform(g, 0.006, 0.015, 1)[0], _uniform(g, 0, 6.28, 1)[0]
        rows.append(a * torch.sin(4.0 * t + p))
    return torch.stack(rows).float().to(DEV).contiguous()


def _gauges_inputs(case, seed):
    g = _generator(seed)
    bed, U = _site(g, case["count"], case["ny"], case["nx"], case["dx"])
    return bed[:, 0].contiguous(), U, _levels(g, case["count"], case["n_out"])


def _inversion_site(case):
    g = _generator(case["ny"] * 1009 + case["batch"])
    bed, U = _site(g, case["batch"], case["ny"], case["nx"], case["dx"])
    return bed, torch.full_like(bed, 0.01), U


def _inversion_inputs(case, seed):
    g = _generator(seed)
    levels = _levels(g, case["batch"], case["n_out"])
    target = _levels(g, case["batch"], case["n_out"])[:, :, None].expand(-1, -1, 6).contiguous()
    return levels, target


def _net_inputs(case, seed):
    g = _generator(seed)
    n = case["batch"]
    t = torch.arange(SAMPLES, dtype=torch.float64) * scenarios.RUNUP_DT_SAMPLE
    x = torch.zeros((n, GAUGES, SAMPLES), dtype=torch.float64)
    for _ in range(4):
        a = (torch.rand((n, GAUGES, 1), generator=g, dtype=torch.float64) - 0.5) * 0.02
        w = torch.rand((n, 1, 1), generator=g, dtype=torch.float64) * 1.5 + 0.2
        p = torch.rand((n, GAUGES, 1), generator=g, dtype=torch.float64) * 6.28
        x += a * torch.sin(w * t + p)
    y = torch.rand((n, CONTROLS), generator=g) * 0.027 - 0.012
    return x.float().to(DEV).contiguous(), normalise_controls(y).to(DEV).contiguous()


def _net_moments(seed, count):
    """Adam's moments in the middle of a training."""
    g = _generator(seed + 1)
    m = torch.randn(count, generator=g) * 3e-4
    v = (torch.rand(count, generator=g) + 0.5) * 1e-6
    return m.to(DEV), v.to(DEV)


MIDDLE_STEP = 400  # Adam steps taken before the timed one

# A program that inverts for an inflow keeps one model of its site and runs
# it again and again; the last site used here is kept the same way.
_sites = {}


def _site_model(case):
    key = tuple(sorted((k, v) for k, v in case.items() if k != "name"))
    if key not in _sites:
        bed, rough, U = _inversion_site(case)
        _sites.clear()
        _sites[key] = (_model(bed, rough, case["dx"], _config("runup"), case["arithmetic"]), U)
    return _sites[key]


# ------------------------------------------------------------ prepare, run
def prepare(case, seed):
    kind = case["kind"]
    s = {"kind": kind, "case": case}
    if kind == "step":
        bed, rough, U, level, rain, infil = _step_inputs(case, seed)
        forcing = RainfallForcing(*rain) if rain is not None else None
        s.update(model=_model(bed, rough, DX, _config(case["sides"], case["friction"]), case["arithmetic"],
                              forcing), U=U, level=level, infil=infil)
    elif kind == "forward":
        bed, rough, U, (times, levels) = _forward_inputs(case, seed)
        model = _model(bed, rough, case["dx"], _config(case["sides"]), case["arithmetic"])
        model.set_dynamic_boundary(times, levels)
        s.update(model=model, U=U)
    elif kind == "ensemble":
        s.update(plan=Ensemble(_ensemble_inputs(case, seed), device=DEV, arithmetic=case["arithmetic"]))
    elif kind == "gauges":
        bed, U, levels = _gauges_inputs(case, seed)
        n = torch.full((1, case["ny"], case["nx"]), 0.01, device=DEV)
        s.update(plan=GaugeEnsemble(bed, n, U, levels, scenarios.RUNUP_DT_SAMPLE,
                                    _gauge_cells(case["ny"], case["nx"]), _config("runup"), case["dx"],
                                    arithmetic=case["arithmetic"]))
    elif kind == "inversion":
        model, U = _site_model(case)
        levels, target = _inversion_inputs(case, seed)
        s.update(model=model, U=U, levels=levels.requires_grad_(True), target=target)
    elif kind == "stepgrad":
        bed, rough, U, level, _, _ = _step_inputs(dict(case, friction="manning", rain=False), seed)
        weight = torch.randn(U.shape, generator=_generator(seed + 1)).to(DEV)
        s.update(model=_model(bed, rough, DX, _config(case["sides"]), case["arithmetic"]),
                 U=U.requires_grad_(True), weight=weight,
                 level=torch.tensor(level, device=DEV, requires_grad=True))
    else:
        net = WarmStartNet(device=DEV, seed=int(seed) % (1 << 31))
        x, y = _net_inputs(case, seed)
        if kind == "train":
            m, v = _net_moments(seed, net.nparams)
            net.m.copy_(m)
            net.v.copy_(v)
            net.step_count = MIDDLE_STEP
        s.update(net=net, x=x, y=y)
    return s


def run(s):
    kind, case = s["kind"], s["case"]
    if kind == "step":
        with torch.no_grad():
            U, dt = s["model"].step(s["U"], model_time=20.0, max_dt=0.02, infiltration=s["infil"],
                                    boundary_level=s["level"])
        return U, dt
    if kind == "forward":
        with torch.no_grad():
            return s["model"](s["U"], t_end=case["t_end"], start_time=1.0)
    if kind == "ensemble":
        return s["plan"].run().states
    if kind == "gauges":
        r = s["plan"].run()
        return r.gauges, r.states
    if kind == "inversion":
        s["levels"].grad = None
        gauges, U = gauge_run(s["model"], s["U"], s["levels"], scenarios.RUNUP_DT_SAMPLE,
                              _gauge_cells(case["ny"], case["nx"]), checkpoint_every=case["every"],
                              store_states=case["store"])
        ((gauges - s["target"]) ** 2).mean(dim=(1, 2)).sum().backward()
        return gauges.detach(), U.detach(), s["levels"].grad
    if kind == "stepgrad":
        s["U"].grad = s["level"].grad = None
        U, dt = s["model"].step(s["U"], model_time=0.0, max_dt=0.02, boundary_level=s["level"])
        (U * s["weight"]).sum().backward()
        return U.detach(), dt, s["U"].grad, s["level"].grad
    if kind == "train":
        loss = s["net"].train_step(s["x"], s["y"])
        return loss, s["net"].grads, s["net"].params
    return s["net"].predict_controls(s["x"])


def work(case):
    """Least bytes and operations of a pass."""
    kind = case["kind"]
    if kind in ("train", "predict"):
        macs = 282 * 32 * 54 + 70 * 64 * 256 + 35 * 128 * 384 + 4480 * 96 + 96 * 96 + 96 * 16
        n, params = case["batch"], 508528
        if kind == "predict":
            return {"bytes": n * (GAUGES * SAMPLES + CONTROLS) * 4 + params * 4, "flops": 2.0 * macs * n}
        return {"bytes": n * (GAUGES * SAMPLES + CONTROLS) * 4 + params * 4 * 7, "flops": 6.0 * macs * n}
    flops = 2.0 * FLOPS_PER_STAGE
    if kind == "step":
        cells = case["ny"] * case["nx"]
        fields = 2 + (3 if case["rain"] else 0)
        return {"bytes": cells * 4 * (6 * case["batch"] + fields), "flops": cells * case["batch"] * flops}
    if kind == "stepgrad":
        cells = case["ny"] * case["nx"]
        return {"bytes": cells * 4 * (15 * case["batch"] + 2), "flops": cells * case["batch"] * 4 * flops}
    if kind == "forward":
        cells, steps = case["ny"] * case["nx"], case["t_end"] / STEP_S
        return {"bytes": cells * steps * 32.0, "flops": cells * steps * flops}
    if kind == "ensemble":
        cells = sum(a * b for a, b in
                    scenarios.ensemble_sizes(case["count"], case["lo"], case["hi"], case["sizes_seed"]))
        return {"bytes": cells * case["steps"] * 32.0, "flops": cells * case["steps"] * flops}
    steps = case["n_out"] * scenarios.RUNUP_DT_SAMPLE / (STEP_S * case["dx"] / DX)
    cells = case["ny"] * case["nx"] * case.get("count", case.get("batch"))
    if kind == "gauges":
        return {"bytes": cells * steps * 32.0, "flops": cells * steps * flops}
    return {"bytes": cells * steps * (32.0 + 56.0), "flops": cells * steps * 4 * flops}


# ---------------------------------------------------------------- 64 bits
# The step in plain torch, float64: B-Flood reconstruction, HLL fluxes and
# semi-implicit friction with the midpoint rule.
def _minmod(a, b, c):
    same = ((a > 0) & (b > 0) & (c > 0)) | ((a < 0) & (b < 0) & (c < 0))
    return torch.where(same, torch.sign(a) * torch.minimum(a.abs(), torch.minimum(b.abs(), c.abs())),
                       torch.zeros_like(a))


class _Exact:
    """A model in float64: bed, rough [1 or B, ny, nx], level a number or [B]."""

    def __init__(self, bed, rough, dx, cfg):
        self.z, self.n, self.dx, self.cfg = bed.double(), rough.double(), float(dx), cfg
        self.floor = max(cfg.epsilon, cfg.dry_depth, 1e-6)
        self.small = max(cfg.epsilon, 1e-6)

    def ghosts(self, U, level, axis):
        """U [B,3,...] and the bed with two ghost lines at both ends of `axis` (-1: x, -2: y)."""
        cfg, n = self.cfg, U.shape[axis]
        codes = ((cfg.boundary_left, cfg.boundary_right) if axis == -1
                 else (cfg.boundary_top, cfg.boundary_bottom))
        Z = self.z[:, None]
        normal = 1 if axis == -1 else 2
        lev = level.reshape(-1, 1, 1, 1) if torch.is_tensor(level) else level
        parts_u, parts_z = [None, None], [None, None]
        for end, code in enumerate(codes):
            edge = 0 if end == 0 else n - 1
            if code == "periodic":
                start = n - 2 if end == 0 else 0
                parts_u[end], parts_z[end] = U.narrow(axis, start, 2), Z.narrow(axis, start, 2)
                continue
            e, ez = U.narrow(axis, edge, 1), Z.narrow(axis, edge, 1)
            rep = torch.cat([e, e], axis)
            parts_z[end] = torch.cat([ez, ez], axis)
            ch = list(rep.split(1, dim=1))
            zz = parts_z[end]
            if code == "water_level":
                ch[0] = torch.clamp(lev - zz, min=0.0).expand_as(ch[0])
            elif code == "wall":
                mirror = U.narrow(axis, 0 if end == 0 else n - 2, 2).flip(axis)
                ch[normal] = -mirror[:, normal:normal + 1]
            elif code == "absorbing":
                hr = torch.clamp(lev - zz, min=0.0).expand_as(ch[0])
                hc = torch.where(hr > 1e-4, hr, ch[0])
                c = torch.sqrt(9.81 * torch.clamp(hc, min=1e-6))
                ch[normal] = (-c if end == 0 else c) * (ch[0] - hr)
            elif code == "constant":
                ch = [torch.full_like(x, cfg.constant_value) for x in ch]
            parts_u[end] = torch.cat(ch, 1)
        return torch.cat([parts_u[0], U, parts_u[1]], axis), torch.cat([parts_z[0], Z, parts_z[1]], axis)

    def direction(self, U, level, axis):
        """Flux difference of the three channels along `axis` and the largest wave speed per member."""
        cfg, g = self.cfg, self.cfg.gravity
        W, z = self.ghosts(U, level, axis)
        z = z[:, 0]
        m = W.shape[axis]

        def at(q, o, count):
            return q.narrow(axis, o, count)

        h = torch.clamp(W[:, 0], min=0.0)
        wet, safe = h > cfg.dry_depth, torch.clamp(h, min=self.floor)
        zero = torch.zeros_like(h)
        u, v = torch.where(wet, W[:, 1] / safe, zero), torch.where(wet, W[:, 2] / safe, zero)
        z = z.expand_as(h)
        eta = h + z

        def inc(q):
            a, c, b = at(q, 0, m - 2), at(q, 1, m - 2), at(q, 2, m - 2)
            return _minmod(cfg.limiter_theta * (c - a), 0.5 * (b - a), cfg.limiter_theta * (b - c))

        dh, de, dz, du, dv = inc(h), inc(eta), inc(z), inc(u), inc(v)
        hc, ec, zc, uc, vc = (at(q, 1, m - 2) for q in (h, eta, z, u, v))
        if cfg.water_slope_reset:
            half, base = 0.5 * (de - dh), ec - hc
            reset = (de * de > dz * dz) & ((base - half > at(eta, 0, m - 2)) | (base + half > at(eta, 2, m - 2)))
            de = torch.where(reset, dh + dz, de)
        q = torch.where(hc > cfg.dry_depth, 0.5 * dh / torch.clamp(hc, min=self.floor), torch.zeros_like(hc))
        fl, fr = torch.clamp(1 - q, -10, 10), torch.clamp(1 + q, -10, 10)
        k = m - 3  # faces
        hL, eL, bL = (at(a + 0.5 * d, 0, k) for a, d in ((hc, dh), (ec, de), (zc, dz)))
        hR, eR, bR = (at(a - 0.5 * d, 1, k) for a, d in ((hc, dh), (ec, de), (zc, dz)))
        uL, vL = at(uc + 0.5 * fl * du, 0, k), at(vc + 0.5 * fl * dv, 0, k)
        uR, vR = at(uc - 0.5 * fr * du, 1, k), at(vc - 0.5 * fr * dv, 1, k)
        b = torch.minimum(torch.maximum(bL, bR), torch.minimum(eL, eR))
        HL = torch.clamp(torch.minimum(eL - b, hL), min=0.0)
        HR = torch.clamp(torch.minimum(eR - b, hR), min=0.0)
        srcL = 0.5 * g * (at(hc, 0, k) + HL) * (at(zc, 0, k) - b)
        srcR = 0.5 * g * (HR + at(hc, 1, k)) * (at(zc, 1, k) - b)

        def prim(H, a, c):
            w, s = H > cfg.dry_depth, torch.clamp(H, min=self.floor)
            o = torch.zeros_like(H)
            return (w, torch.where(w, H * a / s, o), torch.where(w, H * c / s, o),
                    torch.where(w, torch.sqrt(g * s), o))

        wL, uL, vL, cL = prim(HL, uL, vL)
        wR, uR, vR, cR = prim(HR, uR, vR)
        nL, tL, nR, tR = (uL, vL, uR, vR) if axis == -1 else (vL, uL, vR, uR)
        us, cs = 0.5 * (nL + nR) + cL - cR, 0.5 * (cL + cR) + 0.25 * (nL - nR)
        SL = torch.where(wL, torch.minimum(nL - cL, us - cs), nR - 2 * cR)
        SR = torch.where(wR, torch.maximum(nR + cR, us + cs), nL + 2 * cL)
        fhL, fhR = HL * nL, HR * nR
        fqL, fqR = HL * (nL * nL + 0.5 * g * HL), HR * (nR * nR + 0.5 * g * HR)
        den = torch.clamp(SR - SL, min=self.small)
        fh = (SR * fhL - SL * fhR + SL * SR * (HR - HL)) / den
        fq = (SR * fqL - SL * fqR + SL * SR * (fhR - fhL)) / den
        fh = torch.where(SL >= 0, fhL, torch.where(SR <= 0, fhR, fh))
        fq = torch.where(SL >= 0, fqL, torch.where(SR <= 0, fqR, fq))
        any_wet, o = wL | wR, torch.zeros_like(fh)
        fh, fq = torch.where(any_wet, fh, o), torch.where(any_wet, fq, o)
        ft = torch.where(fh > 0, tL, tR) * fh
        speed = torch.where(any_wet, torch.maximum(SL.abs(), SR.abs()), o).detach().amax(dim=(1, 2))
        n = k - 1
        left, right = fq - srcR, fq - srcL

        def diff(lo, hi):
            return (at(lo, 0, n) - at(hi, 1, n)) / self.dx

        return diff(fh, fh), diff(left, right), diff(ft, ft), speed

    def rhs(self, U, level, rain=None, loss=None):
        x0, xn, xt, ax = self.direction(U, level, -1)
        y0, yn, yt, ay = self.direction(U, level, -2)
        r0 = x0 + y0
        if rain is not None:
            r0 = r0 + rain
        if loss is not None:
            r0 = r0 - torch.clamp(loss, min=0.0)
        return torch.stack([r0, xn + yt, xt + yn], 1), ax, ay

    def clean(self, old, new):
        cfg = self.cfg
        if cfg.positivity_limiter:
            d = new - old
            safe = torch.clamp(-d[:, :1], min=cfg.epsilon)
            th = torch.where(d[:, :1] < 0, torch.clamp(old[:, :1] / safe, max=1.0), torch.ones_like(safe))
            new = old + th * d
        h = torch.clamp(new[:, :1], min=0.0)
        q = torch.where(h > cfg.dry_depth, new[:, 1:], torch.zeros_like(new[:, 1:]))
        return torch.cat([h, q], 1)

    def friction(self, U, dt):
        cfg = self.cfg
        if not cfg.apply_friction:
            return U
        h = torch.clamp(U[:, 0], min=0.0)
        wet, safe = h > cfg.dry_depth, torch.clamp(h, min=self.floor)
        o = torch.zeros_like(h)
        u, v = torch.where(wet, U[:, 1], o) / safe, torch.where(wet, U[:, 2], o) / safe
        s2 = u * u + v * v
        speed = torch.where(wet & (s2 > 0), torch.sqrt(torch.clamp(s2, min=self.small ** 2)), o)
        hs = torch.clamp(h, min=self.small)
        if cfg.frictionmodel == "manning":
            cf = 9.81 * torch.clamp(self.n, min=0.0) ** 2 / hs ** (1.0 / 3.0)
        else:
            r = hs / torch.clamp(self.n, min=self.small)
            shallow = 1 / torch.clamp(0.46 * r, min=self.small)
            rc = torch.clamp(r, min=self.small)
            lt = 2.5 * (torch.log(rc) - 1 + 1.359 / rc)
            cf = torch.where(r < math.e, shallow, 1 / torch.clamp(lt * lt, min=self.small))
        f = 1 / (1 + cf * speed * dt / safe)
        return torch.stack([h, torch.where(wet, U[:, 1] * f, o), torch.where(wet, U[:, 2] * f, o)], 1)

    def step(self, U, level, max_dt, rain=None, loss=None, own=False):
        """(new state, dt); own: a time step of its own per member, max_dt [B], else one for all.
        rain: a function of the time since the step's start."""
        k1, ax, ay = self.rhs(U, level, rain(0.0) if rain else None, loss)
        if not own:
            ax, ay = ax.max(), ay.max()
        dt = self.cfg.cfl / torch.clamp(ax / self.dx + ay / self.dx, min=self.cfg.epsilon)
        dt = torch.minimum(dt, torch.as_tensor(max_dt, dtype=torch.float64, device=dt.device))
        d4, d3 = (dt.reshape(-1, 1, 1, 1), dt.reshape(-1, 1, 1)) if own else (dt, dt)
        P = self.clean(U, U + 0.5 * d4 * k1)
        k2, _, _ = self.rhs(P, level, rain(0.5 * float(dt)) if rain else None, loss)
        return self.friction(self.clean(U, U + d4 * k2), d3), dt


def _interpolate(times, levels, t):
    i = min(max(int(torch.searchsorted(times, torch.tensor(t, dtype=times.dtype, device=times.device))), 1),
            times.numel() - 1)
    t0, t1, w0, w1 = (float(x) for x in (times[i - 1], times[i], levels[i - 1], levels[i]))
    return w0 + (t - t0) / (t1 - t0) * (w1 - w0)


def _advance(model, U, duration, level_at, hmax=None):
    elapsed = 0.0
    while duration - elapsed > 1e-12:
        U, dt = model.step(U, level_at(elapsed), duration - elapsed)
        elapsed += float(dt)
        if hmax is not None:
            hmax = torch.maximum(hmax, U[:, 0])
    return U, hmax


def _exact_inversion(case, seed):
    from torch.utils.checkpoint import checkpoint
    bed, rough, U = _inversion_site(case)
    levels, target = _inversion_inputs(case, seed)
    model = _Exact(bed[:, 0], rough[:, 0], case["dx"], _config("runup"))
    lv = levels.double().requires_grad_(True)
    U, cells, rec = U.double(), _gauge_cells(case["ny"], case["nx"]), []
    for i in range(case["n_out"]):
        elapsed = 0.0
        while scenarios.RUNUP_DT_SAMPLE - elapsed > 1e-12:
            U, dt = checkpoint(model.step, U, lv[:, i], scenarios.RUNUP_DT_SAMPLE - elapsed,
                               use_reentrant=False)
            elapsed += float(dt)
        rec.append(torch.stack([U[:, 0, a, b] + model.z[:, a, b] for a, b in cells], -1))
    gauges = torch.stack(rec, 1)
    ((gauges - target.double()) ** 2).mean(dim=(1, 2)).sum().backward()
    return gauges.detach(), U.detach(), lv.grad


def _exact_gauges(case, seed):
    bed, U, levels = _gauges_inputs(case, seed)
    n = torch.full((1, case["ny"], case["nx"]), 0.01, device=DEV)
    model = _Exact(bed, n, case["dx"], _config("runup"))
    U, lv, rec = U.double(), levels.double(), []
    for i in range(case["n_out"]):
        left = torch.full((case["count"],), scenarios.RUNUP_DT_SAMPLE, dtype=torch.float64, device=DEV)
        while bool((left > 1e-12).any()):
            V, dt = model.step(U, lv[:, i], left.clamp(min=1e-9), own=True)
            on = left > 1e-12
            U = torch.where(on.reshape(-1, 1, 1, 1), V, U)
            left = torch.where(on, left - dt, left)
        rec.append(torch.stack([U[:, 0, a, b] + model.z[:, a, b]
                                for a, b in _gauge_cells(case["ny"], case["nx"])], -1))
    return torch.stack(rec, 1), U


def _exact_net(case, seed):
    net = WarmStartNet(device=DEV, seed=int(seed) % (1 << 31))
    p = net.params.double().clone().requires_grad_(True)
    x, y = _net_inputs(case, seed)
    a = x.double() * INPUT_SCALE
    for i, (L, (w, rows, kp, b)) in enumerate(zip(net.layers, net.layout)):
        W, bias = p[w:w + rows * kp].view(rows, kp), p[b:b + rows]
        if isinstance(L, Conv):
            W = W[:, :L.kdim].reshape(rows, L.k, L.cin).transpose(1, 2)
            a = torch.nn.functional.conv1d(a, W, bias, stride=L.stride, padding=L.pad)
        else:
            if a.ndim == 3:
                a = a.transpose(1, 2).reshape(a.shape[0], -1)
            a = a @ W.t() + bias
        if i < 5:
            a = torch.nn.functional.gelu(a)
    if case["kind"] == "predict":
        return (a * CONTROL_SCALE + CONTROL_MEAN).detach()
    loss = ((a - y.double()) ** 2).mean()
    grads, = torch.autograd.grad(loss, p)
    m, v = _net_moments(seed, net.nparams)
    t = MIDDLE_STEP + 1
    m, v = 0.9 * m.double() + 0.1 * grads, 0.999 * v.double() + 0.001 * grads ** 2
    new = p.detach() - 1e-3 * (m / (1 - 0.9 ** t)) / ((v / (1 - 0.999 ** t)).sqrt() + 1e-8)
    return loss.detach().reshape(1), grads, new


def exact(case, seed):
    kind = case["kind"]
    if kind in ("train", "predict"):
        return _exact_net(case, seed)
    if kind == "inversion":
        return _exact_inversion(case, seed)
    if kind == "gauges":
        with torch.no_grad():
            return _exact_gauges(case, seed)
    if kind == "ensemble":
        out = []
        with torch.no_grad():
            for sc in _ensemble_inputs(case, seed):
                model = _Exact(sc.bed[None], sc.roughness[None], sc.dx, SWEConfig(**sc.config))
                U, t = sc.U0.double(), 0.0
                for _ in range(case["steps"]):
                    level = 0.0 if sc.bc_times is None else _interpolate(sc.bc_times, sc.bc_levels, t)
                    U, dt = model.step(U, level, 1e9)
                    t += float(dt)
                out.append(U)
        return out
    if kind == "forward":
        bed, rough, U, (times, levels) = _forward_inputs(case, seed)
        model = _Exact(bed[:, 0], rough[:, 0], case["dx"], _config(case["sides"]))
        with torch.no_grad():
            U = U.double()
            return _advance(model, U, case["t_end"], lambda t: _interpolate(times, levels, 1.0 + t),
                            U[:, 0].clone())
    if kind == "stepgrad":
        bed, rough, U, level, _, _ = _step_inputs(dict(case, friction="manning", rain=False), seed)
        weight = torch.randn(U.shape, generator=_generator(seed + 1)).to(DEV).double()
        model = _Exact(bed[:, 0], rough[:, 0], DX, _config(case["sides"]))
        U = U.double().requires_grad_(True)
        level = torch.tensor(level, device=DEV).double().requires_grad_(True)
        new, dt = model.step(U, level, 0.02)
        gU, gl = torch.autograd.grad((new * weight).sum(), (U, level), allow_unused=True)
        return new.detach(), dt.detach(), gU, torch.zeros_like(level) if gl is None else gl
    bed, rough, U, level, rain, infil = _step_inputs(case, seed)
    model = _Exact(bed[:, 0], rough[:, 0], DX, _config(case["sides"], case["friction"]))

    def rate(after):
        w = (20.0 + after) / 60.0
        return ((1 - w) * rain[1][0] + w * rain[1][1]).double()

    with torch.no_grad():
        new, dt = model.step(U.double(), level, 0.02, rate if rain is not None else None,
                             None if infil is None else infil[:, 0].double())
    return new, dt
