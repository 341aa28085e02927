"""The calls that this framework's performance is judged by, one case per kind of use.

A case is a deck (sizes in voxels of 2.5 um, beam, layers, temperature model) and what a program does with it:

  run       a whole run from the deck to the final state (a small job: launches and per-step latency count)
  steps     a window of the time loop of a developed run, then the state on the host (the framework's main path)
  transfer  the loop driven from the host: the state uploaded, a few steps, the state downloaded
  resume    a checkpoint restored, a few steps, the state on the host
  start     a simulation created, its microstructure generated and first layer laid
  output    the datasets of an output point (SetBuild, temperature, colour maps)
  batch     an ensemble of independent single-track runs, started and run to their ends
  adjoint   melt-pool shape and summed growth of a window and their gradient (a calibration step)

The seed names the realisation (baseplate grains, layer grains, nucleation), so other seeds are other microstructures.
"""
import math
import os
import shutil
import tempfile

import numpy as np
import torch

from amcafe_gb300.adjoint import GrowthRun, Objective
from amcafe_gb300.cafe import Batch, Simulation
from amcafe_gb300.ensemble import deck_text
from amcafe_gb300.rosenthal import pool

DX = 2.5e-6
T_LIQ, T_SOL, T0 = 1609.0, 1531.5, 300.0
ETA, COND, DIFF = 0.35, 20.0, 5e-6  # absorptivity, conductivity, diffusivity of the shipped decks


def listed():
    return [
        # the shipped single-track deck (128x64x32), whole run: the job of a first try and of parameter sweeps
        dict(name="run_single_track", kind="run", nx=128, ny=64, nz=32, speed=1.0, power=200.0, base=4, layer=28,
             hatch=1000.0, scan=0.0, turn=0.0, stride=0.25, nuc=2e-4, mu=1.25e-4, model="pool"),
        # a small ragged part of rotated layers with heavy nucleation, one voxel of beam travel per step, whole run
        dict(name="run_ragged_layers", kind="run", nx=37, ny=29, nz=21, speed=1.0, power=80.0, base=9, layer=6,
             hatch=40.0, scan=2.0, turn=0.7, stride=1.0, nuc=4e-3, mu=4e-4, model="pool"),
        # the shipped four-layer raster (512x256x128) in its developed state
        dict(name="raster_512", kind="steps", nx=512, ny=256, nz=128, speed=1.0, power=200.0, base=80, layer=12,
             hatch=100.0, scan=1.0, turn=0.0, stride=0.25, nuc=2e-4, mu=1.25e-4, model="pool", spin=900, steps=60),
        # the shipped ten-layer rotated build (1024x1024x256, 268 M voxels): the benchmark's workload
        dict(name="build_1024", kind="steps", nx=1024, ny=1024, nz=256, speed=0.8, power=200.0, base=136, layer=12,
             hatch=100.0, scan=2.0, turn=1.1693705988, stride=0.25, nuc=2e-4, mu=2.963e-4, model="pool", spin=1000,
             steps=60),
        # the moving point source's own field (per-cell growth velocities), several tracks of the shipped 256x128x64 box
        dict(name="rosenthal_256", kind="steps", nx=256, ny=128, nz=64, speed=1.0, power=200.0, base=4, layer=20,
             hatch=100.0, scan=1.0, turn=0.0, stride=0.25, nuc=2e-4, mu=1.25e-4, model="rosenthal", spin=400, steps=20),
        # the EASM temperature (a numerical integral per cell and step), box sides no powers of two
        dict(name="easm_odd", kind="steps", nx=181, ny=93, nz=47, speed=1.0, power=200.0, base=4, layer=20,
             hatch=100.0, scan=1.0, turn=0.0, stride=0.25, nuc=2e-4, mu=1.25e-4, model="easm", spin=120, steps=20),
        # the loop coupled to a host program: upload, ten steps, download
        dict(name="host_coupled_512", kind="transfer", nx=512, ny=256, nz=128, speed=1.0, power=200.0, base=80,
             layer=12, hatch=100.0, scan=1.0, turn=0.0, stride=0.25, nuc=2e-4, mu=1.25e-4, model="pool", spin=800,
             steps=10),
        # a job continued from its checkpoint
        dict(name="resume_256", kind="resume", nx=256, ny=256, nz=128, speed=1.0, power=200.0, base=80, layer=12,
             hatch=100.0, scan=1.0, turn=0.0, stride=0.25, nuc=2e-4, mu=1.25e-4, model="pool", spin=800, steps=20),
        # the beginning of every run: grains of the baseplate and of the first layer
        dict(name="start_512", kind="start", nx=512, ny=256, nz=128, speed=1.0, power=200.0, base=80, layer=12,
             hatch=100.0, scan=1.0, turn=0.0, stride=0.25, nuc=2e-4, mu=1.25e-4, model="pool"),
        # what is written at an output point
        dict(name="output_256", kind="output", nx=256, ny=256, nz=128, speed=1.0, power=200.0, base=80, layer=12,
             hatch=100.0, scan=1.0, turn=0.0, stride=0.25, nuc=2e-4, mu=1.25e-4, model="pool", spin=60),
        # parameter studies: independent runs with their own boxes, beams and seeds
        dict(name="ensemble_12", kind="batch", count=12, lo=48, hi=80, boxes=1),
        # a calibration step: values and gradient over a window of the shipped adjoint deck's box
        dict(name="adjoint_256", kind="adjoint", nx=256, ny=128, nz=64, speed=1.0, power=200.0, base=4, layer=60,
             hatch=1000.0, scan=0.0, turn=0.0, stride=0.25, nuc=2e-4, mu=1.25e-4, model="rosenthal", spin=400,
             steps=48),
    ]


def _log(rng, lo, hi):
    """A whole number from lo..hi, even over its logarithm, odd ones among them."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["run", "run", "steps", "steps", "steps", "transfer", "resume", "start", "output", "batch",
                       "adjoint"])
    if kind == "batch":
        lo = _log(rng, 36, 56)
        return dict(kind=kind, count=rng.randint(3, 12), lo=lo, hi=lo + rng.randint(8, 24), boxes=rng.randint(2, 10**6))
    c = dict(kind=kind, speed=round(rng.uniform(0.5, 1.5), 3), power=round(rng.uniform(120.0, 260.0), 1),
             nuc=round(math.exp(rng.uniform(math.log(1e-4), math.log(2e-3))), 7),
             mu=round(rng.uniform(1e-4, 4e-4), 7), turn=0.0, scan=1.0, stride=0.25, hatch=100.0, model="pool")
    if kind == "run":
        c.update(nx=_log(rng, 24, 44), ny=_log(rng, 20, 34), nz=_log(rng, 16, 24), base=rng.randint(4, 8),
                 layer=rng.randint(5, 8), hatch=round(rng.uniform(40.0, 80.0), 1), scan=rng.choice([1.0, 2.0]),
                 stride=rng.choice([0.5, 1.0]), power=round(rng.uniform(60.0, 120.0), 1))
        if c["scan"] == 2.0:
            c["turn"] = round(rng.uniform(0.2, 1.4), 4)
    elif kind == "adjoint":
        c.update(nx=_log(rng, 200, 256), ny=_log(rng, 80, 128), nz=64, base=4, layer=60, hatch=1000.0, scan=0.0,
                 model="rosenthal", spin=350, steps=rng.randint(16, 48), speed=1.0)
    else:
        c.update(nx=_log(rng, 240, 640), ny=_log(rng, 120, 320), nz=_log(rng, 96, 160), base=60, layer=12)
        if kind != "start":
            c["spin"] = rng.randint(700, 900) if kind != "output" else 60
        if kind == "steps":
            c["model"] = rng.choice(["pool", "pool", "pool", "rosenthal", "easm"])
            c["steps"] = rng.randint(20, 60)
            if c["model"] == "rosenthal":
                c.update(nx=_log(rng, 200, 300), ny=_log(rng, 100, 150), nz=64, base=4, layer=20, spin=400, steps=20)
            elif c["model"] == "easm":
                c.update(nx=_log(rng, 150, 200), ny=_log(rng, 80, 110), nz=48, base=4, layer=20, spin=120, steps=16)
            elif rng.random() < 0.5:
                c.update(turn=round(rng.uniform(0.2, 1.4), 4), scan=2.0)
        elif kind in ("transfer", "resume"):
            c["steps"] = rng.randint(4, 24)
    return c


def _deck(case, seed, folder):
    """The case's deck as a file (the shipped decks' keywords and physics)."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    v, power = case["speed"], case["power"]
    front, rear, width, depth = pool(power, v, ETA, COND, DIFF, T_LIQ, T0)
    gy = 0.0 if case["scan"] == 0.0 else case["scan"] * ny * DX
    lines = [
        "dx %r" % DX, "nX %d %d %d" % (nx, ny, nz), "bmV %r" % v, "bmP %r" % power,
        "bmDelT %r" % (case["stride"] * DX / v), "r %r" % case["nuc"], "lT %r" % (case["layer"] * DX),
        "bpH %r" % (case["base"] * DX), "tL %r" % T_LIQ, "tS %r" % T_SOL,
        "meltparam %r %r %r %r" % (front, rear, width, depth), "bhatch %r" % (case["hatch"] * 1e-6),
        "mu %r" % case["mu"], "lrate %r" % case["mu"], "patternID %d" % (1 if gy == 0.0 else 2), "outint 1000000",
        "offset 0.0 0.0 0.0", "gridsize %r %r" % (max(case["scan"], 1.0) * nx * DX, gy),
        "gridtheta %r" % case["turn"], "dendritegrowth2 1e-5 2.0", "seed %d" % (1 + seed % 100003),
    ]
    if case["model"] == "easm":
        lines.append("easm 1")
    if case["model"] == "rosenthal":
        lines += ["rosenthal %r %r %r" % (ETA, COND, DIFF), "nucgauss 7.0 0.5"]
    path = os.path.join(folder, "case.in")
    with open(path, "w") as f:
        f.write("\n".join(lines) + "\n")
    return path


_FIELDS = dict(gID=(1, torch.int32), vState=(1, torch.int32), extents=(1, torch.float64),
               centroid=(3, torch.float64), buildj=(1, torch.int32))
_buffers = {}


def _host_buffers(ncell):
    """Pinned output buffers, kept by a program for all its states of one size."""
    if ncell not in _buffers:
        _buffers.clear()
        _buffers[ncell] = {k: torch.empty(m * ncell, dtype=dt, pin_memory=True) for k, (m, dt) in _FIELDS.items()}
    return _buffers[ncell]


def _state_of(sim, buffers=None):
    if buffers is None:
        return {k: torch.from_numpy(a) for k, a in sim.state().items()}
    sim.state(out={k: b.numpy() for k, b in buffers.items()})
    return dict(buffers)


class _Folder:
    """A temporary folder, removed with the state that uses it."""

    def __init__(self):
        self.path = tempfile.mkdtemp(prefix="cafe_case_")

    def __del__(self):
        shutil.rmtree(self.path, ignore_errors=True)


def prepare(case, seed):
    kind, folder = case["kind"], _Folder()
    state = dict(kind=kind, folder=folder, case=case)
    if kind == "batch":
        state["decks"] = []
        boxes = np.random.default_rng(case["boxes"])  # the study's boxes; beams and grains come from the seed
        beams = np.random.default_rng(seed)
        for k in range(case["count"]):
            path = os.path.join(folder.path, "run%d.in" % k)
            with open(path, "w") as f:
                f.write(deck_text(1 + (seed * 16 + k) % 100003, boxes.integers(case["lo"], case["hi"] + 1, 3),
                                  float(beams.uniform(0.5, 1.5)), float(beams.uniform(150.0, 300.0)), 7.0))
            state["decks"].append(path)
        return state
    deck = state["deck"] = _deck(case, seed, folder.path)
    if kind in ("run", "start"):
        if kind == "start":
            state["out"] = _host_buffers(case["nx"] * case["ny"] * case["nz"])
        return state
    if kind == "adjoint":
        state["grow"] = GrowthRun(deck, case["steps"], spinup=case["spin"], workdir=folder.path)
        # a calibration's current estimate, a little off the run's own parameters
        r = np.random.default_rng(seed)
        th = state["grow"].theta * (1.0 + 0.05 * r.uniform(-1.0, 1.0, 5) * np.array([1, 1, 0, 1, 0]))
        state["theta"] = torch.tensor(th, dtype=torch.float64)
        state["weight"] = torch.tensor([1.0, 0.7, 1.3, 0.4], dtype=torch.float64)
        return state
    sim = state["sim"] = Simulation(deck)
    sim.InitializeVoxels()
    sim.begin()
    sim.run(case["spin"])
    if kind != "output":
        state["out"] = _host_buffers(sim.ncell)
    if kind == "transfer":  # the host program's own copy, updated in place by every pass
        state["out"] = {k: torch.empty(m * sim.ncell, dtype=dt, pin_memory=True) for k, (m, dt) in _FIELDS.items()}
        _state_of(sim, state["out"])
        state["ctheta"] = sim.ctheta()
    if kind == "resume":
        state["checkpoint"] = os.path.join(folder.path, "resume.ckpt")
        sim.checkpoint(state["checkpoint"])
    return state


def run(state):
    kind, case = state["kind"], state["case"]
    if kind == "run":
        with Simulation(state["deck"]) as sim:
            sim.InitializeVoxels()
            sim.begin()
            sim.run()
            return _state_of(sim)
    if kind == "start":
        with Simulation(state["deck"]) as sim:
            sim.InitializeVoxels()
            sim.begin()
            return _state_of(sim, state["out"])
    if kind == "batch":
        with Batch(state["decks"]) as batch:
            batch.run()
            return [_state_of(s) for s in batch.sims]
    if kind == "adjoint":
        theta = state["theta"].clone().requires_grad_(True)
        out = Objective.apply(theta, state["grow"])
        (out * state["weight"]).sum().backward()
        out = out.detach()
        return dict(pool=out[:3], growth=out[3:], grad=theta.grad)
    sim = state["sim"]
    if kind == "output":
        sim.SetBuild()
        return dict({k: torch.from_numpy(a) for k, a in sim.output().items()}, build=torch.from_numpy(sim.build()))
    if kind == "transfer":
        h = {k: b.numpy() for k, b in state["out"].items()}
        sim.upload_state(h["gID"], h["vState"], h["extents"], h["centroid"], state["ctheta"])
    if kind == "resume":
        sim.restore(state["checkpoint"])
    sim.run(case["steps"])
    out = _state_of(sim, state["out"])
    if kind == "transfer":
        state["ctheta"] = sim.ctheta()
    return out


def _pool_cells(case):
    """Cells of the box around the melt pool, clipped to the part."""
    front, rear, width, depth = pool(case["power"], case["speed"], ETA, COND, DIFF, T_LIQ, T0)
    return (min(case["nx"], (front + rear) / DX) * min(case["ny"], 2 * width / DX) * min(case["nz"], depth / DX))


def work(case):
    """Bytes: the voxel fields read once (38 a voxel in the device layout) and written once in the layout that the
    call returns (44 on the host), and one read and write of the states in the pool's box per step."""
    kind = case["kind"]
    if kind == "batch":
        side = (case["lo"] + case["hi"]) / 2
        cells, steps = case["count"] * side ** 3, 4 * side
        return {"bytes": cells * (38 + 44) + case["count"] * steps * 2 * side ** 3 / 4, "flops": 0}
    cells = case["nx"] * case["ny"] * case["nz"]
    box = _pool_cells(case)
    if kind == "run":
        tracks = 1 if case["scan"] == 0.0 else math.ceil(case["ny"] * DX / (case["hatch"] * 1e-6))
        layers = max(1, (case["nz"] - case["base"]) // case["layer"])
        steps = case["nx"] / case["stride"] * tracks * layers
        return {"bytes": cells * (38 + 44) + steps * 2 * box, "flops": 0}
    if kind == "start":
        return {"bytes": cells * (38 + 44), "flops": 0}
    if kind == "output":
        return {"bytes": cells * (4 + 1 + 44), "flops": 0}
    if kind == "adjoint":
        # forward and backward: the field of every cell of every step twice, ~60 operations each
        return {"bytes": 2 * cells * 38, "flops": 2 * (case["steps"] + 1) * cells * 60.0}
    if kind == "transfer":
        return {"bytes": cells * (44 + 38 + 44) + case["steps"] * 2 * box, "flops": 0}
    flops = 0.0
    if case["model"] != "pool":  # the field of every cell below the laser plane: one exponential, or two integrals of 25
        flops = case["steps"] * (case["base"] + case["layer"]) * case["nx"] * case["ny"] * \
            (40.0 if case["model"] == "rosenthal" else 50 * 40.0)
    return {"bytes": cells * (38 + 44) + case["steps"] * 2 * box, "flops": flops}


def exact(case, seed):
    """The melt-pool extents of the adjoint case from their definition; the rest is the automaton's own chain of events."""
    if case["kind"] != "adjoint":
        return None
    r = np.random.default_rng(seed)
    off = 1.0 + 0.05 * r.uniform(-1.0, 1.0, 5) * np.array([1, 1, 0, 1, 0])
    power, eta, v = case["power"] * off[0], ETA * off[1], case["speed"]
    dt = case["stride"] * DX / case["speed"]
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    x, y, z = ((torch.arange(n, dtype=torch.float64, device=dev) + 0.5) * DX for n in (case["nx"], case["ny"], case["nz"]))
    z_src = (case["base"] + case["layer"]) * DX
    z = z[z <= z_src]
    # the source starts at the first point of its track and moves one stride a step; the last logged step is spin + steps
    xs = v * dt * (case["spin"] + case["steps"])
    xi, dy, dz = (x - xs)[None, None, :], (y - case["ny"] * DX / 2)[None, :, None], (z - z_src)[:, None, None]
    R = torch.sqrt(xi * xi + dy * dy + dz * dz).clamp(min=0.5 * DX)
    T = T0 + eta * power / (2 * math.pi * COND) / R * torch.exp(-v * (R + xi) / (2 * DIFF))
    m = torch.sigmoid((T - T_LIQ) / 10.0)
    s = m.sum()

    def mean(f):
        return (m * f).sum() / s

    X, Y = x[None, None, :], y[None, :, None]
    out = torch.stack([torch.sqrt(12 * (mean(X * X) - mean(X) ** 2)), torch.sqrt(12 * (mean(Y * Y) - mean(Y) ** 2)),
                       torch.sqrt(3 * mean(dz * dz))])
    return dict(pool=out.cpu(), growth=None, grad=None)
