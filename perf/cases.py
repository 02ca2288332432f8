"""Workloads of the proton pencil-beam framework, as a treatment-planning
program runs them: the CT's water-equivalent depth, the dose of a plan, its
gradients, a batch of plans and the whole host call.

Every case is a plain dict.  `listed` gives the fixed ones, `draw` further
ones of the same ranges, `prepare` makes a case's inputs from a seed, `run`
is one pass through the public entry points, `work` the bytes and operations
of a pass, and `exact` the same results in 64 bits, from plain torch.

Kinds
  wet        HU -> RLSP -> water-equivalent depth of every beam
             (engine.rlsp_from_hu, DevicePlan.compute_wet)
  dose       dose of all beams from the depths (DevicePlan.forward)
  adjoint    spot-weight gradient of a dose field (DevicePlan.adjoint)
  positions  spot-weight and spot-position gradients
             (DevicePlan.adjoint_positions)
  step       one optimiser step's dose, objective and weight gradient through
             autograd (autograd.dose, autograd.quadratic_objective)
  batch      depths and doses of several uneven plans (batch.BatchPlans.run)
  plan       IMPTDoseGrid.computeIMPTPlan, host CT in, host doses out
"""
from __future__ import annotations

import copy
import functools
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.getcwd(), "dosecuda-jax_b200")
if _PKG not in sys.path:
    sys.path.insert(1, _PKG)

MACHINE = "HitachiProbeatJHU"
SPACINGS = (1.0, 1.5, 2.0, 2.5, 3.0)


def _case(kind, nx, ny, nz, spacing, gantry, couch=0.0, noise=0.0, target=30.0, pitch=5.0,
          layers=10, model=0, **more):
    """gantry: the beams' angles as "0,90" (degrees); noise: HU noise of the
    CT (0: a piecewise-constant phantom); target: mean radius (mm); pitch:
    spot lattice (mm); layers: energies per beam; model: 0 without, 1 with
    the 4 cm range shifter."""
    return dict(kind=kind, nx=nx, ny=ny, nz=nz, spacing=float(spacing), gantry=gantry,
                couch=float(couch), noise=float(noise), target=float(target),
                pitch=float(pitch), layers=layers, model=model, **more)


def listed():
    return [
        # a small CT at a coarse grid with one oblique, couch-rotated beam: what
        # an interactive beam-angle change recomputes
        dict(_case("wet", 96, 88, 72, 3.0, "33.3", couch=15.0, noise=12.0, target=25.0,
                   mode="texture"), name="wet_small"),
        # the benchmark's grid, four beams along the image axes, a phantom
        # without noise (commissioning and QA plans)
        dict(_case("wet", 256, 256, 160, 2.0, "0,90,180,270", target=42.0, mode="texture"),
             name="wet_phantom"),
        # a patient CT: image noise everywhere, a 2.5 mm planning grid
        dict(_case("wet", 200, 188, 160, 2.5, "0,115,241.5", noise=14.0, target=42.0,
                   mode="texture"), name="wet_ct"),
        # exact trilinear depths of a patient CT (the mode for studies that
        # compare with other dose engines)
        dict(_case("wet", 165, 150, 121, 2.0, "70,200", noise=14.0, target=30.0, mode="exact"),
             name="wet_exact"),
        # the smallest plan: one beam, a few layers, a few hundred spots
        dict(_case("dose", 56, 48, 40, 3.0, "45", target=13.0, pitch=5.0, layers=6),
             name="dose_small"),
        # the water cube of the tests: 120^3 at 2.5 mm, 10 layers, ~1,200 spots
        dict(_case("dose", 120, 120, 120, 2.5, "0", target=28.0, pitch=5.0, layers=10),
             name="dose_cube"),
        # the 1 mm optimisation grid: the largest dose, ~60,000 spots on a 3 mm lattice
        dict(_case("dose", 512, 512, 200, 1.0, "0,90,180,270", target=48.0, pitch=3.0, layers=17),
             name="dose_large"),
        # gradient of a small plan on a ragged grid (one field of a robust
        # optimisation, range shifter in)
        dict(_case("adjoint", 101, 93, 77, 2.5, "20,290", target=24.0, pitch=5.0, layers=9,
                   model=1), name="adjoint_small"),
        # weight and position gradients together (spot-position optimisation)
        dict(_case("positions", 128, 121, 88, 2.5, "60,180", target=30.0, pitch=5.0, layers=12),
             name="positions"),
        # one optimiser step of the benchmark's plan: 4 beams, ~20,000 spots
        dict(_case("step", 256, 256, 160, 2.0, "0,90,180,270", target=43.0, pitch=5.0, layers=17),
             name="step_plan"),
        # eight uneven plans in one batch (a robustness or beam-angle study)
        dict(_case("batch", 152, 146, 121, 2.5, "10,140", noise=10.0, target=32.0, pitch=5.0,
                   layers=10, plans=8), name="batch"),
        # the reference's call: host CT in, host doses out, 3 beams, ~8,000 spots
        dict(_case("plan", 256, 256, 160, 2.0, "0,120,240", noise=10.0, target=34.0, pitch=5.0,
                   layers=14), name="plan_host"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("wet", "wet", "wet", "dose", "dose", "dose", "adjoint", "adjoint",
                       "positions", "step", "step", "batch", "plan"))
    top = {"batch": 150, "positions": 170}.get(kind, 256)
    while True:
        spacing = rng.choice(SPACINGS)
        nx, ny, nz = _log(rng, 40, top), _log(rng, 40, top), _log(rng, 36, min(top, 180))
        low = min(nx, ny, nz) * spacing
        if low >= 96.0 and max(nx, ny, nz) * spacing <= 560.0:
            break
    beams = rng.randint(1, 4)
    if rng.random() < 0.35:
        angles = rng.sample((0, 90, 180, 270), beams)
        couch = 0.0
    else:
        angles = [round(rng.uniform(0.0, 360.0), 1) for _ in range(beams)]
        couch = rng.choice((0.0, 0.0, 10.0, 345.0, 90.0))
    target = min(45.0, rng.uniform(0.12, 0.2) * low)
    more = {}
    if kind == "wet":
        more["mode"] = rng.choice(("texture", "texture", "exact"))
    if kind == "batch":
        more["plans"] = rng.randint(2, 8)
    return _case(kind, nx, ny, nz, spacing, ",".join("%g" % a for a in angles), couch=couch,
                 noise=rng.choice((0.0, 5.0, 12.0, 25.0)), target=round(target, 1),
                 pitch=rng.choice((3.5, 5.0, 6.0)), layers=rng.randint(3, 16),
                 model=rng.choice((0, 0, 0, 1)), **more)


# ------------------------------------------------------------------ inputs

def _device():
    return torch.device("cuda", 0)


@functools.lru_cache(maxsize=None)
def _machine():
    """The machine's beam models (read once, as a planning program does)."""
    from dosecuda_b200.plan_impt import IMPTPlan
    return IMPTPlan(MACHINE)


@functools.lru_cache(maxsize=None)
def _curve():
    """The machine's HU -> RLSP curve."""
    import dosecuda_b200
    path = os.path.join(os.path.dirname(dosecuda_b200.__file__), "lookuptables", "protons",
                        MACHINE, "HU_RLSP.csv")
    t = np.genfromtxt(path, delimiter=",", names=True)
    return np.ascontiguousarray(t["HU"], np.float64), np.ascontiguousarray(t["RLSP"], np.float64)


def _interp(hu):
    """numpy.interp of HU over the curve, in 64 bits on hu's device."""
    xh, yh = (torch.as_tensor(a, device=hu.device) for a in _curve())
    x = hu.double()
    j = (torch.searchsorted(xh, x, right=True) - 1).clamp_(0, len(xh) - 2)
    f = ((x - xh[j]) / (xh[j + 1] - xh[j])).clamp_(0.0, 1.0)
    return yh[j] + f * (yh[j + 1] - yh[j])


class _Frame:
    """A beam's geometry in 64 bits: isocentre relative to the first voxel,
    source and the rotation between the image and the beam's-eye frame."""

    def __init__(self, gantry, couch, iso, origin, model):
        ga = math.radians(math.fmod(gantry + 180.0, 360.0))
        ta = math.radians(couch)
        sg, cg, st, ct = math.sin(ga), math.cos(ga), math.sin(ta), math.cos(ta)
        self.iso = np.asarray(iso, np.float64) - np.asarray(origin, np.float64)
        self.vx, self.vy = float(model.VSADX), float(model.VSADY)
        self.sad = 0.5 * (self.vx + self.vy)
        # rows: image (x, y, z) -> head (x, y, z)
        self.R = np.array([[-ct * cg, -sg, st * cg], [st, 0.0, ct], [-ct * sg, cg, st * sg]])
        self.src = self.R.T @ np.array([0.0, 0.0, self.sad])

    def head(self, x, y, z):
        """Head-frame coordinates of image points relative to the isocentre."""
        r = self.R
        return tuple(r[a, 0] * x + r[a, 1] * y + r[a, 2] * z for a in range(3))


def _voxels(frame, shape, spacing, dtype=torch.float64):
    """Image coordinates (mm, relative to the isocentre) of every voxel."""
    nz, ny, nx = shape
    ax = [torch.arange(n, device=_device(), dtype=dtype) * spacing - float(frame.iso[a])
          for a, n in enumerate((nx, ny, nz))]
    return ax[0][None, None, :], ax[1][None, :, None], ax[2][:, None, None]


def _scene(case, seed):
    """CT, beams and spots of a case: water in air with bone and lung slabs
    and spheres, image noise, an ellipsoidal target off the voxel lattice,
    per beam a spot lattice over the target's projection and energies across
    its depth."""
    rng = np.random.default_rng([int(seed), 977])
    dev = _device()
    s = case["spacing"]
    n = (case["nx"], case["ny"], case["nz"])
    shape = (n[2], n[1], n[0])
    ext = np.array(n) * s
    origin = (-0.5 * ext).astype(np.float32)
    hu = torch.full(shape, -1000.0, device=dev)
    m = max(1, int(round(10.0 / s)))
    hu[m:-m, m:-m, m:-m] = 0.0
    ax = [torch.arange(k, device=dev, dtype=torch.float32) * s + float(o)
          for k, o in zip(n, origin)]

    def cut(a, lo, hi):
        lo, hi = sorted((int((lo - origin[a]) / s), int((hi - origin[a]) / s)))
        return slice(max(lo, m), max(min(hi, n[a] - m), m))

    for q in range(9):
        c = rng.uniform(-0.36, 0.36, 3) * ext
        value = 1000.0 if rng.random() < 0.5 else -700.0
        if q < 3:   # slab
            half = rng.uniform(0.08, 0.22, 3) * ext
            half[rng.integers(3)] = rng.uniform(4.0, 14.0)
            sl = [cut(a, c[a] - half[a], c[a] + half[a]) for a in range(3)]
            hu[sl[2], sl[1], sl[0]] = value
        else:       # sphere
            r = rng.uniform(0.03, 0.08) * ext.min()
            sl = [cut(a, c[a] - r, c[a] + r) for a in range(3)]
            d2 = ((ax[2][sl[2]] - c[2]) ** 2)[:, None, None] + \
                ((ax[1][sl[1]] - c[1]) ** 2)[None, :, None] + \
                ((ax[0][sl[0]] - c[0]) ** 2)[None, None, :]
            hu[sl[2], sl[1], sl[0]] = torch.where(d2 <= r * r, value, hu[sl[2], sl[1], sl[0]])
    if case["noise"] > 0.0:
        g = torch.Generator(device=dev)
        g.manual_seed(int(seed) * 7919 + 13)
        hu += case["noise"] * torch.randn(shape, device=dev, generator=g)
        hu.clamp_(min=-1024.0)

    semi = case["target"] * rng.uniform(0.85, 1.15, 3)
    centre = rng.uniform(-0.06, 0.06, 3) * ext + rng.uniform(0.1, 0.9, 3) * s
    iso = centre.astype(np.float32)
    target = (((ax[0] - centre[0]) / semi[0]) ** 2)[None, None, :] + \
        (((ax[1] - centre[1]) / semi[1]) ** 2)[None, :, None] + \
        (((ax[2] - centre[2]) / semi[2]) ** 2)[:, None, None] <= 1.0

    plan = copy.copy(_machine())
    plan.beam_list, plan.n_beams = [], 0
    model = plan.beam_models[case["model"]]
    frames = []
    for angle in (float(a) for a in case["gantry"].split(",")):
        f = _Frame(angle, case["couch"], iso, origin, model)
        # water-equivalent depth of the target's centre: samples every mm
        # along the central axis
        step = torch.arange(0.0, float(np.linalg.norm(ext)), 1.0, device=dev)
        at = [((step * float(f.src[a] / f.sad) + float(f.iso[a])) / s).round().long()
              for a in range(3)]
        ok = (at[0] >= 0) & (at[0] < n[0]) & (at[1] >= 0) & (at[1] < n[1]) & \
            (at[2] >= 0) & (at[2] < n[2])
        depth = float(_interp(hu[at[2][ok], at[1][ok], at[0][ok]]).clamp(min=0.0).sum())
        axis = f.R[2]
        reach = float(np.sqrt(np.sum((semi * axis) ** 2)))
        # energies across the target's depth, evenly over the machine's table
        # (the same number of layers and spots whatever the seed)
        r80 = model.divergence_params[:, 1].astype(np.float64)
        usable = np.flatnonzero(r80 >= 30.0)
        ends = [int(np.argmin(np.abs(r80[usable] - d)))
                for d in (depth - reach, depth + 1.05 * reach)]
        short = max(0, case["layers"] - 1 - (ends[1] - ends[0]))
        lo = min(max(0, ends[0] - short // 2), len(usable) - case["layers"])
        hi = min(max(ends[1], lo + case["layers"] - 1), len(usable) - 1)
        ids = usable[np.round(np.linspace(lo, hi, case["layers"])).astype(int)]
        # lattice over the target's projection, 3 mm margin
        k = int(math.ceil((case["target"] + 3.0) / case["pitch"]))
        lat = np.arange(-k, k + 1) * case["pitch"]
        X, Y = (a.ravel() for a in np.meshgrid(lat, lat, indexing="ij"))
        inside = X * X + Y * Y <= (case["target"] + 3.0) ** 2
        xy = np.stack([X[inside], Y[inside]], axis=1)
        spots = np.concatenate([np.column_stack([xy, rng.uniform(0.5, 1.5, len(xy)),
                                                 np.full(len(xy), e)]) for e in ids[::-1]])
        from dosecuda_b200.plan_impt import IMPTBeam
        beam = IMPTBeam()
        beam.dicom_rangeshifter_label = str(plan.dicom_rangeshifter_label[case["model"]])
        beam.gantry_angle, beam.couch_angle = angle, case["couch"]
        beam.iso = iso.copy()
        beam.spot_list = np.ascontiguousarray(spots, np.float32)
        beam.n_spots = len(spots)
        plan.addBeam(beam)
        frames.append(f)
    return dict(hu=hu, shape=shape, spacing=s, origin=origin, iso=iso, plan=plan, model=model,
                frames=frames, target=target, semi=semi, centre=centre)


def _depths(sc):
    """Water-equivalent depth (cm) of every voxel and beam, as an earlier pass
    over the CT left it: marched on a grid of half the resolution, then
    interpolated (beams x voxels, float32)."""
    s = sc["spacing"]
    rlsp = _interp(sc["hu"]).float()
    vol = rlsp[None, None]
    nz, ny, nx = sc["shape"]
    n = (nx, ny, nz)
    out = torch.empty((len(sc["frames"]), nz * ny * nx), device=_device())
    coarse = tuple((k + 1) // 2 for k in (nz, ny, nx))
    for b, f in enumerate(sc["frames"]):
        # coarse points at voxel coordinates spread over the whole grid
        p = []
        for a, (k, m) in enumerate(zip(n, reversed(coarse))):
            p.append(torch.linspace(0.0, k - 1.0, m, device=_device()) * s - float(f.iso[a]))
        p = [p[0][None, None, :].expand(coarse), p[1][None, :, None].expand(coarse),
             p[2][:, None, None].expand(coarse)]
        u = [float(f.src[a]) - p[a] for a in range(3)]
        inv = torch.rsqrt(u[0] ** 2 + u[1] ** 2 + u[2] ** 2)
        # normalised grid_sample coordinates and their step of 2 mm
        at = torch.stack([((p[a] + float(f.iso[a])) / s + 0.5) * 2.0 / n[a] - 1.0
                          for a in range(3)], -1)[None]
        step = torch.stack([u[a] * inv * (4.0 / (s * n[a])) for a in range(3)], -1)[None]
        wet = torch.zeros(coarse, device=_device())
        for _ in range(int(0.5 * s * math.sqrt(nx * nx + ny * ny + nz * nz)) + 1):
            wet += torch.nn.functional.grid_sample(vol, at, align_corners=False)[0, 0]
            at += step
        wet = 0.2 * wet - 0.1
        out[b] = torch.nn.functional.interpolate(wet[None, None], size=sc["shape"],
                                                 mode="trilinear",
                                                 align_corners=True).reshape(-1)
    return out


def _specs(sc):
    from dosecuda_b200 import engine
    return [engine.BeamSpec(b.gantry_angle, b.couch_angle, b.iso, b.spot_list, sc["model"])
            for b in sc["plan"].beam_list]


def _device_plan(sc):
    from dosecuda_b200 import engine
    return engine.DevicePlan(sc["shape"], sc["spacing"], sc["origin"], _specs(sc), _device())


def _objective(sc):
    """Prescription 60 in the target, 0 outside; voxel weights 1 / 0.1."""
    presc = torch.where(sc["target"], 60.0, 0.0).reshape(-1)
    weight = torch.where(sc["target"], 1.0, 0.1).reshape(-1)
    return presc, weight


def _field(sc, seed):
    """d objective / d dose: signed values in and around the target, zero
    farther away."""
    g = torch.Generator(device=_device())
    g.manual_seed(int(seed) * 104729 + 5)
    z = torch.randn(sc["shape"], device=_device(), generator=g)
    r2 = 0.0
    for a, view in zip(range(3), ((None, None, slice(None)), (None, slice(None), None),
                                  (slice(None), None, None))):
        n = sc["shape"][2 - a]
        x = torch.arange(n, device=_device(), dtype=torch.float32) * sc["spacing"] + \
            float(sc["origin"][a])
        r2 = r2 + (((x - float(sc["centre"][a])) / (2.0 * float(sc["semi"][a]))) ** 2)[view]
    return torch.where(r2 < 2.0, z * torch.exp(-r2), 0.0).reshape(-1)


def _sub_cases(case):
    """The uneven plans of a batch."""
    rng = np.random.default_rng([case["nx"], case["ny"], case["nz"], 31])
    subs = []
    for p in range(case["plans"]):
        f = rng.uniform(0.55, 1.0, 3) if p else np.ones(3)
        sub = dict(case, kind="dose")
        sub.update(nx=int(case["nx"] * f[0]), ny=int(case["ny"] * f[1]), nz=int(case["nz"] * f[2]),
                   target=float(case["target"] * f.min()),
                   layers=max(2, int(case["layers"] * rng.uniform(0.5, 1.0))))
        if p % 3 == 2:
            sub["gantry"] = case["gantry"].split(",")[0]
        subs.append(sub)
    return subs


def prepare(case, seed):
    from dosecuda_b200 import engine
    kind = case["kind"]
    if kind == "batch":
        from dosecuda_b200 import batch
        plans, rlsps = [], []
        for p, sub in enumerate(_sub_cases(case)):
            sc = _scene(sub, int(seed) * 131 + p)
            dp = _device_plan(sc)
            rlsp = engine.rlsp_from_hu(sc["hu"].reshape(-1), *_curve())
            dp.compute_wet(rlsp)
            plans.append(dp)
            rlsps.append(rlsp)
        return dict(kind=kind, batch=batch.BatchPlans(plans, rlsps))
    sc = _scene(case, seed)
    if kind == "plan":
        from dosecuda_b200.plan_impt import IMPTDoseGrid
        grid = IMPTDoseGrid()
        grid.origin = sc["origin"].astype(np.float64)
        grid.spacing = np.full(3, sc["spacing"])
        grid.size = np.array(sc["shape"])
        grid.HU = sc["hu"].cpu().numpy()
        return dict(kind=kind, grid=grid, plan=sc["plan"])
    dp = _device_plan(sc)
    if kind == "wet":
        return dict(kind=kind, plan=dp, hu=sc["hu"].reshape(-1), mode=case["mode"])
    dp.set_wet(_depths(sc))
    state = dict(kind=kind, plan=dp)
    if kind in ("adjoint", "positions"):
        state["field"] = _field(sc, seed)
    if kind == "step":
        state["presc"], state["weight"] = _objective(sc)
        state["mu"] = dp.mu_plan().clone()
    return state


def run(state):
    kind = state["kind"]
    if kind == "batch":
        b = state["batch"]
        b.run()
        return {"dose": b.doses, "wet": [dp.wet for dp in b.plans]}
    if kind == "plan":
        g = state["grid"]
        g.computeIMPTPlan(state["plan"])
        return {"dose": g.dose, "beams": g.beam_doses, "rlsp": g.RLSP}
    dp = state["plan"]
    if kind == "wet":
        from dosecuda_b200 import engine
        rlsp = engine.rlsp_from_hu(state["hu"], *_curve())
        return {"rlsp": rlsp, "wet": dp.compute_wet(rlsp, wet_mode=state["mode"])}
    if kind == "dose":
        return dp.forward()
    if kind == "adjoint":
        return dp.to_plan(dp.adjoint(state["field"]))
    if kind == "positions":
        return tuple(dp.to_plan(g) for g in dp.adjoint_positions(state["field"]))
    from dosecuda_b200 import autograd
    mu = state["mu"].clone().requires_grad_(True)
    dose = autograd.dose(mu, dp)
    objective = autograd.quadratic_objective(dose, state["presc"], state["weight"])
    objective.backward()
    return {"dose": dose.detach(), "objective": objective.detach(), "grad": mu.grad}


def work(case):
    """Each input read and each output written once.  A depth sample is one
    trilinear interpolation per mm of the mean path out of the grid (half the
    shorter lateral extent), with 54 additions of the lateral smoothing; a
    spot reaches the voxels within 60 mm of its axis (where its halo is above
    2^-24 of its peak) over 0.7 of the grid's mean extent, 12 operations
    each."""
    if case["kind"] == "batch":
        parts = [work(sub) for sub in _sub_cases(case)]
        wets = [work(dict(sub, kind="wet")) for sub in _sub_cases(case)]
        return {k: sum(p[k] for p in parts) + sum(w[k] for w in wets) for k in ("bytes", "flops")}
    V = case["nx"] * case["ny"] * case["nz"]
    s = case["spacing"]
    ext = sorted((case["nx"] * s, case["ny"] * s, case["nz"] * s))
    B = len(case["gantry"].split(","))
    per_layer = math.pi * (case["target"] + 3.0) ** 2 / case["pitch"] ** 2
    S = B * per_layer * case["layers"]
    radius = min(60.0, 0.5 * ext[0])
    dose_flops = S * math.pi * radius ** 2 * 0.7 * ext[1] / s ** 3 * 12.0
    wet_flops = B * V * (0.5 * ext[1] * 20.0 + 54.0)
    dose_bytes = 4.0 * V * (B + 1) + 36.0 * S
    wet_bytes = 4.0 * V * (2 + B)
    return {"wet": {"bytes": wet_bytes, "flops": wet_flops},
            "dose": {"bytes": dose_bytes, "flops": dose_flops},
            "adjoint": {"bytes": dose_bytes, "flops": dose_flops},
            "positions": {"bytes": dose_bytes, "flops": 3.0 * dose_flops},
            "step": {"bytes": 2.0 * dose_bytes + 12.0 * V, "flops": 2.0 * dose_flops},
            "plan": {"bytes": 4.0 * V * (3 + 2 * B), "flops": wet_flops + dose_flops},
            }[case["kind"]]


# --------------------------------------------------------- 64-bit results

def _exact_depths(sc, rlsp):
    """Smoothed water-equivalent depth (cm) with exact trilinear samples."""
    nz, ny, nx = sc["shape"]
    s = sc["spacing"]
    n = (nx, ny, nz)
    # one layer of zeros around the volume: the border of the interpolation
    pad = torch.zeros((nz + 2, ny + 2, nx + 2), device=_device(), dtype=torch.float64)
    pad[1:-1, 1:-1, 1:-1] = rlsp
    flat = pad.reshape(-1)
    sy, sz = nx + 2, (nx + 2) * (ny + 2)
    out = []
    for f in sc["frames"]:
        p = [c.expand(sc["shape"]).reshape(-1) for c in _voxels(f, sc["shape"], s)]
        u = [float(f.src[a]) - p[a] for a in range(3)]
        inv = 1.0 / torch.sqrt(u[0] ** 2 + u[1] ** 2 + u[2] ** 2)
        u = [c * inv for c in u]
        total = torch.zeros(nx * ny * nz, device=_device(), dtype=torch.float64)
        live = torch.arange(nx * ny * nz, device=_device())
        for t in range(int(s * math.sqrt(nx * nx + ny * ny + nz * nz)) + 3):
            x = [(p[a] + u[a] * t + float(f.iso[a])) / s + 0.5 for a in range(3)]
            ok = torch.ones_like(live, dtype=torch.bool)
            for a in range(3):
                ok &= (x[a] >= 0.0) & (x[a] < n[a])
            if not bool(ok.all()):
                live, x = live[ok], [c[ok] for c in x]
                p, u = [c[ok] for c in p], [c[ok] for c in u]
            if live.numel() == 0:
                break
            lo = [torch.floor(c - 0.5) for c in x]
            w = [c - 0.5 - l for c, l in zip(x, lo)]
            base = (lo[0] + 1 + sy * (lo[1] + 1) + sz * (lo[2] + 1)).long()
            v = 0.0
            for q in range(8):
                wx = w[0] if q & 1 else 1.0 - w[0]
                wy = w[1] if q & 2 else 1.0 - w[1]
                wz = w[2] if q & 4 else 1.0 - w[2]
                v = v + wx * wy * wz * flat[base + (q & 1) + sy * ((q >> 1) & 1) + sz * (q >> 2)]
            total[live] += v.clamp(min=0.0)
        raw = 0.1 * total - 0.05
        x, y, z = _voxels(f, sc["shape"], s)
        h = [c.expand(sc["shape"]).reshape(-1) for c in f.head(x, y, z)]
        limit = 10.0 * raw
        acc, count = raw.clone(), torch.ones_like(raw)
        for d in range(6):
            for r in range(1, 10):
                hx, hy = h[0] + r * math.cos(d * math.pi / 3), h[1] + r * math.sin(d * math.pi / 3)
                idx, ok = 0, limit > r
                for a, stride in zip(range(3), (1, nx, nx * ny)):
                    q = f.R[0, a] * hx + f.R[1, a] * hy + f.R[2, a] * h[2] + float(f.iso[a])
                    q = torch.floor(q / s + 0.5).long()
                    ok = ok & (q >= 0) & (q < n[a])
                    idx = idx + q.clamp(0, n[a] - 1) * stride
                acc += torch.where(ok, raw[idx], 0.0)
                count += ok
        out.append(torch.where(limit > 1.0, acc / count, raw))
    return torch.stack(out)


def _layers(spots):
    """(energy id, rows of the spot list) of each layer."""
    ids = spots[:, 3].astype(int)
    return [(e, np.flatnonzero(ids == e)) for e in sorted(set(ids.tolist()))]


def _influence(sc, wet):
    """Yields (beam, spot rows, voxel indexes, x, y, weight per unit spot) over
    the plan: a function of the spots' x and y gives the dose of a unit weight
    at those voxels (voxels x spots, 64 bits)."""
    model = sc["model"]
    s = sc["spacing"]
    for b, f in enumerate(sc["frames"]):
        spots = np.asarray(sc["plan"].beam_list[b].spot_list)
        w32 = wet[b] * 10.0
        depth = wet[b].double() * 10.0
        X, Y, Z = (c.expand(sc["shape"]).reshape(-1)
                   for c in f.head(*_voxels(f, sc["shape"], s)))
        for e, rows in _layers(spots):
            r80 = float(model.divergence_params[e, 1])
            ca, cb, cc = (float(v) for v in model.divergence_params[e, 2:5])
            cut = float(np.float32(1.1) * np.float32(r80))
            gx, gy = 1.0 - Z / f.vx, 1.0 - Z / f.vy
            # voxels in range and within 130 mm of the layer's spot box (its
            # Gaussians are below 1e-20 of their peak farther out)
            box = [torch.stack([q * g for q in (v.min(), v.max())])
                   for v, g in ((spots[rows, 0], gx), (spots[rows, 1], gy))]
            dx = torch.relu(torch.maximum(box[0].amin(0) - X, X - box[0].amax(0)))
            dy = torch.relu(torch.maximum(box[1].amin(0) - Y, Y - box[1].amax(0)))
            at = torch.nonzero((w32 <= cut) & (dx * dx + dy * dy < 130.0 ** 2))[:, 0]
            del dx, dy, box
            lut = [torch.as_tensor(np.asarray(t[e], np.float64), device=_device())
                   for t in (model.lut_depths, model.lut_sigmas, model.lut_idds)]
            chunk = max(1, (1 << 25) // len(rows))
            for c in range(0, at.numel(), chunk):
                v = at[c:c + chunk]
                yield b, rows, v, _unit_dose(f, X[v], Y[v], Z[v], depth[v], r80, ca, cb, cc, lut)


def _unit_dose(f, X, Y, Z, wet, r80, ca, cb, cc, lut):
    dep, sig, idd = lut
    lo = torch.searchsorted(dep, wet)
    hi, lo = lo.clamp(0, len(dep) - 1), (lo - 1).clamp(min=0)
    gap = dep[hi] - dep[lo]
    t = torch.where((gap > 0) & (wet <= dep[-1]), (wet - dep[lo]) / torch.where(gap > 0, gap, 1.0),
                    1.0).clamp(0.0, 1.0)
    i0 = idd[lo] + t * (idd[hi] - idd[lo])
    mcs = sig[lo] + t * (sig[hi] - sig[lo])
    dist = torch.sqrt(X * X + Y * Y + (f.sad - Z) ** 2)
    d = dist - wet + 0.7 * r80
    st2 = (ca * d * d + cb * d + cc + mcs) ** 2
    w = wet.clamp(min=0.1).clamp(max=r80 - 0.1)
    sh = 2.85 + 0.0014 * r80 * torch.log(w + 3.0) + 0.06 * w - 7.4e-5 * w * w - \
        0.22 * r80 / (w - r80 - 5.0) ** 2
    wh = 0.052 * torch.log(1.13 + w / (11.2 - 0.023 * r80)) + \
        0.35 * (0.0017 * r80 * r80 - r80) / ((r80 + 3.0) ** 2 - w * w) - \
        1.61e-9 * w * (r80 + 3.0) ** 2
    sh, wh = sh.clamp(min=0.0), wh.clamp(0.0, 0.9)
    sht2 = st2 + sh * sh
    pf = (1.0 - wh) * i0 / (2.0 * math.pi * st2)
    hf = wh * i0 / (2.0 * math.pi * sht2)

    def at(xs, ys):
        tx, ty = xs / f.vx, ys / f.vy
        gx, gy = 1.0 - Z / f.vx, 1.0 - Z / f.vy
        # |t x ray|^2 / |t|^2 of the spot's diverging axis
        q = (X[:, None] - gx[:, None] * xs) ** 2
        q = q + (Y[:, None] - gy[:, None] * ys) ** 2
        q = q + (Y[:, None] * tx - X[:, None] * ty - xs * ys * (1.0 / f.vx - 1.0 / f.vy)) ** 2
        q = q / (1.0 + tx * tx + ty * ty)
        return pf[:, None] * torch.exp(q * (-0.5 / st2)[:, None]) + \
            hf[:, None] * torch.exp(q * (-0.5 / sht2)[:, None])
    return at


def _columns(sc):
    """x, y, weight of every beam's spots (64 bits, on the device)."""
    return [[torch.as_tensor(np.asarray(b.spot_list)[:, q].astype(np.float64), device=_device())
             for q in range(3)] for b in sc["plan"].beam_list]


def _exact_dose(sc, wet):
    dose = torch.zeros(wet.shape[1], device=_device(), dtype=torch.float64)
    cols = _columns(sc)
    for b, rows, v, at in _influence(sc, wet):
        x, y, mu = (c[rows] for c in cols[b])
        dose[v] += at(x, y) @ mu
    return dose


def _exact_gradient(sc, wet, field):
    cols = _columns(sc)
    grads = [torch.zeros_like(c[0]) for c in cols]
    for b, rows, v, at in _influence(sc, wet):
        wv = field[v]
        if not bool((wv != 0).any()):
            continue
        grads[b][rows] += at(cols[b][0][rows], cols[b][1][rows]).T @ wv
    return torch.cat(grads)


def _exact_positions(sc, wet, field):
    cols = _columns(sc)
    grads = [[torch.zeros_like(c[0]) for _ in range(3)] for c in cols]
    for b, rows, v, at in _influence(sc, wet):
        v_at = field[v] != 0
        if not bool(v_at.any()):
            continue
        x, y, mu = (c[rows].clone().requires_grad_(True) for c in cols[b])
        torch.dot(field[v], at(x, y) @ mu).backward()
        for g, t in zip(grads[b], (mu, x, y)):
            g[rows] += t.grad
    return tuple(torch.cat([g[q] for g in grads]) for q in range(3))


def exact(case, seed):
    kind = case["kind"]
    if kind == "batch":
        return None            # depths sampled by the texture unit have no 64-bit value
    V = case["nx"] * case["ny"] * case["nz"]
    if kind in ("dose", "adjoint", "positions", "step"):
        # spot-voxel pairs of a few 1e11 take some ten seconds
        pairs = work(case)["flops"] / 12.0
        if pairs * case["spacing"] > 1.2e11:
            return None
    sc = _scene(case, seed)
    rlsp = _interp(sc["hu"])
    if kind == "plan":
        return {"dose": None, "beams": [None] * len(sc["frames"]), "rlsp": rlsp}
    if kind == "wet":
        if case["mode"] == "texture" or V * len(sc["frames"]) > 2.5e7:
            return {"rlsp": rlsp.reshape(-1), "wet": None}
        # the depths are those of the float32 RLSP that the pass works on
        return {"rlsp": rlsp.reshape(-1), "wet": _exact_depths(sc, rlsp.float().double())}
    wet = _depths(sc)
    if kind == "dose":
        return _exact_dose(sc, wet)
    if kind == "adjoint":
        return _exact_gradient(sc, wet, _field(sc, seed).double())
    if kind == "positions":
        return _exact_positions(sc, wet, _field(sc, seed).double())
    dose = _exact_dose(sc, wet)
    presc, weight = (t.double() for t in _objective(sc))
    miss = dose - presc
    return {"dose": dose, "objective": (weight * miss * miss).sum(),
            "grad": _exact_gradient(sc, wet, 2.0 * weight * miss)}
