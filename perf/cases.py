"""The work a user of this package has it do, as cases that can be timed and compared.

Each case names a ``kind`` of work and its sizes; ``prepare`` makes what a user's program
holds before the call (meshes, solvers, tracers, beams, fields), ``run`` makes one pass
through the package's public entry points, ``work`` says what such a pass cannot do
without and ``exact`` gives its outputs from plain torch in 64 bits where that is quick.

The kinds: the kernel catalogue's gather and deposit; the field solves (linear, Boltzmann
plasma, refined boxes); the traces (Runge-Kutta and Boris, in a magnetic field, in 3D);
the reverse sweep of a trace, which every design gradient is made of; and whole solves
(a small diode, the einzel lens, a batch of candidate lenses).
"""

from __future__ import annotations

import math
from dataclasses import replace

import numpy as np
import torch

import beamtracer_b200 as bt
from beamtracer_b200.adjoint import TraceAdjoint
from beamtracer_b200.batch import BatchedVlasov
from beamtracer_b200.einzel import EinzelDesign, einzel_config, sweep_designs
from beamtracer_b200.fields import MeshArrays, StaggeredElectricField
from beamtracer_b200.geometry3d import (
    BeamTracer3D,
    Electrode3D,
    IonOpticsMesh3D,
    StaggeredElectricField3D,
)
from beamtracer_b200.kernels import KERNELS
from beamtracer_b200.model import BeamOptics, config_particles
from beamtracer_b200.poisson import BoltzmannElectrons, IonOpticsPoisson
from beamtracer_b200.refinement import Refinement
from beamtracer_b200.solenoid_extraction import SolenoidExtractionDesign, solenoid_extraction

MM = 1e-3
EPS0 = 8.8541878188e-12
CHARGE = 1.602176634e-19
PROTON = 1.67262192e-27
#: The refined extraction's boxes: (level, lower, upper) over the aperture.
BOXES = ((1, (0.0, 0.0), (2.0 * MM, 1.5 * MM)), (2, (0.0, 0.0), (1.5 * MM, 1.2 * MM)))


def listed() -> list[dict]:
    return [
        # the field at every trajectory's position, as a host-driven tracer asks for it at
        # each of its stages: the smallest call there is
        {"name": "gather", "kind": "gather", "nx": 401, "ny": 101, "points": 20_011},
        # a step's charges of a large beam added to the lens's mesh
        {"name": "deposit", "kind": "deposit", "nx": 801, "ny": 201, "points": 1_000_003,
         "cylindrical": True},
        # one Vlasov iteration's field of the einzel lens
        {"name": "field_lens", "kind": "field", "ny": 201},
        # one iteration's Newton solve of the plasma extraction, graded along x
        {"name": "field_plasma", "kind": "plasma", "nx": 1025, "ny": 513},
        # the same on the composite mesh of an extraction with boxes over its aperture
        {"name": "field_refined", "kind": "refined", "nx": 81, "ny": 31, "boxes": 2,
         "plasma": True},
        # one iteration's trace of the lens's rings, deposit included
        {"name": "trace_lens", "kind": "trace", "ny": 201, "rings": 20_000,
         "integrator": "rk4"},
        # one iteration's trace of the plasma extraction's beam in its solenoid
        {"name": "trace_magnetic", "kind": "magnetic", "nx": 1025, "ny": 513,
         "trajectories": 100_000},
        # a beam through a 3D gap with a plate
        {"name": "trace_3d", "kind": "trace3d", "cells": 40, "trajectories": 100_000,
         "integrator": 0, "magnetic": False, "current": False},
        # the reverse of a trace: what a design gradient repeats
        {"name": "adjoint_sweep", "kind": "adjoint", "ny": 101, "rings": 8_000},
        # the smallest whole solve: the planar diode
        {"name": "diode_run", "kind": "diode", "nx": 41, "ny": 21, "trajectories": 40},
        # the headline: the einzel lens from its configuration to its moments
        {"name": "lens_run", "kind": "lens", "ny": 201, "rings": 20_000},
        # a design sweep's candidates converged together
        {"name": "sweep_run", "kind": "sweep", "candidates": 16},
    ]  # fmt: skip


def _log(rng, low: int, high: int) -> int:
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng) -> dict:
    kind = rng.choice(["gather", "deposit", "field", "plasma", "refined", "trace", "trace",
                       "magnetic", "trace3d", "adjoint", "diode", "lens", "sweep"])  # fmt: skip
    if kind == "gather":
        return {"kind": kind, "nx": _log(rng, 41, 801), "ny": _log(rng, 21, 201),
                "points": _log(rng, 100, 4_000_000)}  # fmt: skip
    if kind == "deposit":
        return {"kind": kind, "nx": _log(rng, 41, 1025), "ny": _log(rng, 21, 257),
                "points": _log(rng, 1_000, 4_000_000), "cylindrical": rng.random() < 0.5}  # fmt: skip
    if kind == "field":
        return {"kind": kind, "ny": rng.randint(41, 201)}
    if kind == "plasma":
        return {"kind": kind, "nx": _log(rng, 129, 1025), "ny": _log(rng, 65, 513)}
    if kind == "refined":
        k = rng.randint(1, 2)
        return {"kind": kind, "nx": 80 * k + 1, "ny": 30 * k + 1, "boxes": rng.randint(1, 2),
                "plasma": rng.random() < 0.5}  # fmt: skip
    if kind == "trace":
        return {"kind": kind, "ny": rng.randint(41, 201), "rings": _log(rng, 200, 20_000),
                "integrator": rng.choice(["rk4", "boris"])}  # fmt: skip
    if kind == "magnetic":
        return {"kind": kind, "nx": _log(rng, 129, 1025), "ny": _log(rng, 65, 513),
                "trajectories": _log(rng, 400, 100_000)}  # fmt: skip
    if kind == "trace3d":
        return {"kind": kind, "cells": rng.randint(12, 40),
                "trajectories": _log(rng, 500, 100_000), "integrator": rng.randint(0, 1),
                "magnetic": rng.random() < 0.5, "current": rng.random() < 0.25}  # fmt: skip
    if kind == "adjoint":
        return {"kind": kind, "ny": rng.randint(41, 101), "rings": _log(rng, 500, 8_000)}
    if kind == "diode":
        k = rng.randint(10, 60)
        return {"kind": kind, "nx": 2 * k + 1, "ny": k + 1,
                "trajectories": _log(rng, 40, 1_000)}  # fmt: skip
    if kind == "lens":
        return {"kind": kind, "ny": rng.randint(51, 201), "rings": _log(rng, 500, 20_000)}
    return {"kind": kind, "candidates": rng.randint(2, 14)}


# -- what a program holds before the call --------------------------------------------------------


def _smooth(generator, shape):
    """A seeded smooth array of the shape, values about 1: a few long waves."""
    axes = [torch.linspace(0.0, 1.0, n, dtype=torch.float64, device="cuda") for n in shape]
    grid = torch.meshgrid(*axes, indexing="ij")
    out = torch.ones(shape, dtype=torch.float64, device="cuda")
    for _ in range(4):
        c = torch.rand(len(shape) + 1, generator=generator, dtype=torch.float64)
        out += 0.2 * torch.sin(sum(6.0 * float(c[a]) * g for a, g in enumerate(grid))
                               + 6.28 * float(c[-1]))  # fmt: skip
    return out


def _lens_design(case: dict, seed: int) -> EinzelDesign:
    ny = case["ny"]
    return EinzelDesign(shape=(4 * (ny - 1) + 1, ny), trajectories=case.get("rings", 1_000),
                        seed=seed)  # fmt: skip


def _beam_density(mesh, generator, radius: float, scale: float):
    """A beam's charge density on a mesh's nodes: a core of the radius with seeded waves."""
    r = torch.from_numpy(np.array(mesh.y)).cuda()[None, :]
    return scale * _smooth(generator, mesh.shape) * torch.exp(-((r / radius) ** 2))


def _lens_tracer(case: dict, seed: int, integrator: str = "rk4") -> dict:
    """The lens's mesh and tracer with its beam loaded, and the vacuum field's edges."""
    model = BeamOptics(einzel_config(_lens_design(case, seed), integrator=integrator))
    mesh = model.mesh
    phi = torch.zeros(mesh.shape, dtype=torch.float64, device="cuda")
    IonOpticsPoisson(mesh).solve_device(phi)
    electric = StaggeredElectricField(mesh, phi)
    engine = model.tracer.engine()
    engine.load(config_particles(model.config)[0])
    return {"mesh": mesh, "engine": engine, "fx": electric.fx_device, "fy": electric.fy_device}


def _diode_config(case: dict, seed: int):
    neumann = bt.FieldBoundaryCondition.neumann(0.0)
    volts = -1000.0 - 10.0 * (seed % 17)
    beam = bt.BeamSpecies("H+", 10.0, (0.0, 0.0), (0.0, 5 * MM), energy=0.01,
                          transverse_temperature=0.0, num_particles=case["trajectories"])  # fmt: skip
    return bt.BeamOpticsConfig(
        grid=bt.GridParams(ndim=2, num_gridpoints=(case["nx"], case["ny"]),
                           lower_bound=(0.0, 0.0), upper_bound=(10 * MM, 5 * MM),
                           coordinates="cartesian"),
        bcs_field=bt.FieldBCs(bt.FieldBoundaryCondition.dirichlet(0.0),
                              bt.FieldBoundaryCondition.dirichlet(volts), neumann, neumann),
        beams=[beam], diagnostic_planes=[9.9 * MM], iterations=20, tolerance=1e-3,
        relaxation=1.0,
    )  # fmt: skip


def _extraction_config(case: dict):
    """Ions extracted through a round aperture from a plasma, cylindrical."""
    def plate(x0, x1, r0, voltage):
        return bt.ObjectParams(type="aperture2d", axis=0, position=0.0,
                               vertices=((x0, r0), (x0, 3.1 * MM), (x1, 3.1 * MM), (x1, r0)),
                               bc_type="dirichlet", bc_value=voltage)  # fmt: skip

    neumann = bt.FieldBoundaryCondition.neumann(0.0)
    return bt.BeamOpticsConfig(
        grid=bt.GridParams(ndim=2, num_gridpoints=(case["nx"], case["ny"]),
                           lower_bound=(0.0, 0.0), upper_bound=(8 * MM, 3 * MM),
                           coordinates="cylindrical"),
        bcs_field=bt.FieldBCs(bt.FieldBoundaryCondition.dirichlet(5.0),
                              bt.FieldBoundaryCondition.dirichlet(-2000.0), neumann, neumann),
        objects={"pg": plate(0.5 * MM, 1.0 * MM, 1.0 * MM, 0.0),
                 "eg": plate(3.0 * MM, 4.0 * MM, 1.2 * MM, -2000.0)},
        beams=[bt.BeamSpecies("ion", 50.0, (0.0, 0.0), (0.0, 0.9 * MM), charge=1.0, mass=1.0,
                              energy=5.0, transverse_temperature=0.5, num_particles=100)],
        iterations=2, tolerance=1e-4,
    )  # fmt: skip


def _plasma_design(case: dict, seed: int) -> SolenoidExtractionDesign:
    return replace(SolenoidExtractionDesign(), shape=(case["nx"], case["ny"]), seed=seed,
                   trajectories=case.get("trajectories", 100))  # fmt: skip


def prepare(case: dict, seed: int) -> dict:
    kind = case["kind"]
    g = torch.Generator().manual_seed(seed)
    on_gpu = torch.Generator(device="cuda").manual_seed(seed)
    f64 = dict(dtype=torch.float64, device="cuda")
    state: dict = {"kind": kind}
    if kind in ("gather", "deposit"):
        nx, ny, n = case["nx"], case["ny"], case["points"]
        h = 20.0 * MM / (ny - 1)
        state |= {"h": h, "px": torch.rand(n, generator=on_gpu, **f64) * h * (nx - 1),
                  "py": torch.rand(n, generator=on_gpu, **f64) ** 2 * h * (ny - 1)}  # fmt: skip
        if kind == "gather":
            state |= {"fx": 1e6 * _smooth(g, (nx + 1, ny)), "fy": 1e6 * _smooth(g, (nx, ny + 1)),
                      "ex": torch.empty(n, **f64), "ey": torch.empty(n, **f64)}  # fmt: skip
        else:
            state |= {"q": 1e-16 * (0.5 + torch.rand(n, generator=on_gpu, **f64)),
                      "cylindrical": case["cylindrical"], "charge": torch.zeros((nx, ny), **f64)}  # fmt: skip
    elif kind == "field":
        mesh = BeamOptics(einzel_config(_lens_design(case, seed))).mesh
        state |= {"mesh": mesh, "solver": IonOpticsPoisson(mesh),
                  "rho": _beam_density(mesh, g, 2 * MM, 3e-5),
                  "phi": torch.zeros(mesh.shape, **f64)}  # fmt: skip
    elif kind == "plasma":
        design = _plasma_design(case, seed)
        mesh = solenoid_extraction(design).mesh
        y = torch.from_numpy(np.array(mesh.y)).cuda()[None, :] - design.axis_y
        x = torch.from_numpy(np.array(mesh.x)).cuda()[:, None]
        # the extracted sheet: thinning as the ions speed up
        rho = (9e-3 * _smooth(g, mesh.shape) * torch.exp(-((y / (1.5 * MM)) ** 6))
               / torch.sqrt(1.0 + (x / MM) ** 2))  # fmt: skip
        solver = IonOpticsPoisson(mesh)
        first = torch.zeros(mesh.shape, **f64)
        solver.solve_device(first, None, fixed_region=lambda x, y: x < design.plasma_x,
                            fixed_potential=design.plasma_potential)  # fmt: skip
        species = BoltzmannElectrons(CHARGE * design.electron_density,
                                     design.electron_temperature, design.plasma_potential)  # fmt: skip
        state |= {"mesh": mesh, "solver": solver, "rho": rho, "first": first,
                  "phi": torch.empty(mesh.shape, **f64), "species": species}  # fmt: skip
    elif kind == "refined":
        mesh = BeamOptics(_extraction_config(case)).mesh
        boxes = [Refinement(*box) for box in BOXES[: case["boxes"]]]
        solver = IonOpticsPoisson(mesh, refinement=boxes)
        x, r = (torch.from_numpy(a).cuda() for a in solver.coordinates)
        c = torch.rand(3, generator=g, dtype=torch.float64)
        waves = 1.0 + 0.3 * torch.sin(800.0 * float(c[0]) * x + 900.0 * float(c[1]) * r + float(c[2]))
        rho = 1.5e-3 * waves * torch.exp(-((r / (0.8 * MM)) ** 4)) / torch.sqrt(1.0 + (x / MM) ** 2)
        first = torch.zeros(rho.shape, **f64)
        solver.solve_device(first, None, fixed_region=lambda x, y: x < 0.6 * MM,
                            fixed_potential=5.0)  # fmt: skip
        species = BoltzmannElectrons(1.6e-3, 5.0, 5.0) if case["plasma"] else None
        state |= {"solver": solver, "rho": rho, "first": first, "phi": torch.empty_like(first),
                  "species": species}  # fmt: skip
    elif kind == "trace":
        state |= _lens_tracer(case, seed, case["integrator"])
    elif kind == "magnetic":
        design = _plasma_design(case, seed)
        built = solenoid_extraction(design)
        phi = torch.zeros(built.mesh.shape, **f64)
        IonOpticsPoisson(built.mesh).solve_device(
            phi, None, fixed_region=lambda x, y: x < design.plasma_x,
            fixed_potential=design.plasma_potential)  # fmt: skip
        electric = StaggeredElectricField(built.mesh, phi)
        engine = built.tracer.engine()
        engine.load(built.particles)
        state |= {"mesh": built.mesh, "engine": engine, "design": design,
                  "field": built.magnetic.field, "fx": electric.fx_device,
                  "fy": electric.fy_device}  # fmt: skip
    elif kind == "trace3d":
        state |= _prepare_3d(case, g, on_gpu)
    elif kind == "adjoint":
        state |= _lens_tracer(case, seed)
        engine = state["engine"]
        engine.run(state["fx"], state["fy"])
        hits = torch.randn(engine.hits.shape, generator=on_gpu, **f64)
        hits[..., 1:3] *= 1e-2
        hits[..., 3:6] *= 1e-8
        state |= {"adjoint": TraceAdjoint(engine, state["fx"], state["fy"]),
                  "charge_seed": 1e6 * _smooth(g, state["mesh"].shape), "hit_seed": hits}  # fmt: skip
    elif kind == "diode":
        state["config"] = _diode_config(case, seed)
    elif kind == "lens":
        state["config"] = einzel_config(_lens_design(case, seed))
    elif kind == "sweep":
        # the sweep's candidates, each seed with its own voltages, currents and beams
        scale = np.random.default_rng(seed).uniform(0.95, 1.05, (case["candidates"], 2))
        designs = [replace(d, voltages=(0.0, float(d.voltages[1] * v), 0.0),
                           current=float(d.current * c), seed=d.seed + 1000 * seed)
                   for d, (v, c) in zip(sweep_designs(case["candidates"]), scale)]  # fmt: skip
        state["configs"] = [einzel_config(d, iterations=20) for d in designs]
    else:
        raise ValueError(f"unknown kind {kind!r}")
    return state


def _prepare_3d(case: dict, g, on_gpu) -> dict:
    """A beam through a gap 4 times as long as wide with a plate holding a round aperture."""
    m, n = case["cells"], case["trajectories"]
    h = 20.0 * MM / m
    f64 = dict(dtype=torch.float64, device="cuda")
    half = 10.0 * MM

    def inside(x, y, z):
        on_plate = (x >= 38.0 * MM) & (x <= 42.0 * MM)
        return on_plate & ((y - half) ** 2 + (z - half) ** 2 >= (6.0 * MM) ** 2)

    mesh = IonOpticsMesh3D((4 * m + 1, m + 1, m + 1), (0.0, 0.0, 0.0), h,
                           [Electrode3D(inside, 2000.0)])  # fmt: skip
    x, y, z = (torch.from_numpy(a).cuda() for a in mesh.nodes())
    phi = 50.0 * _smooth(g, mesh.shape) - 3e4 * x + 2000.0 * torch.exp(-(((x - 40 * MM) / (9 * MM)) ** 2))
    phi = phi + 3e6 * ((y - half) ** 2 + (z - half) ** 2) * torch.exp(-(((x - 40 * MM) / (7 * MM)) ** 2))
    fixed = torch.from_numpy(mesh.fixed).cuda()
    phi = torch.where(fixed, torch.from_numpy(mesh.fixed_value).cuda(), phi)
    electric = StaggeredElectricField3D(mesh, phi)
    cells, subcells = BeamTracer3D(mesh, electric).electrode_lookup()
    radius = 4.0 * MM * torch.sqrt(torch.rand(n, generator=on_gpu, **f64))
    angle = 6.283185307179586 * torch.rand(n, generator=on_gpu, **f64)
    x0 = torch.stack([torch.full((n,), 0.5 * MM, **f64), half + radius * torch.cos(angle),
                      half + radius * torch.sin(angle)])  # fmt: skip
    speed = 1.0e6
    v0 = torch.stack([speed * (1.0 + 0.01 * torch.randn(n, generator=on_gpu, **f64)),
                      5e-3 * speed * torch.randn(n, generator=on_gpu, **f64),
                      5e-3 * speed * torch.randn(n, generator=on_gpu, **f64)])  # fmt: skip
    nodes = int(np.prod(mesh.shape))
    ints = dict(dtype=torch.int64, device="cuda")
    magnetic = torch.zeros((3, 2, 2, 2), **f64)
    if case["magnetic"]:
        magnetic = torch.stack([0.05 * _smooth(g, mesh.shape), 0.002 * _smooth(g, mesh.shape),
                                0.002 * _smooth(g, mesh.shape)]).contiguous()  # fmt: skip
    return {
        "mesh": mesh, "electric": electric, "cells": torch.from_numpy(cells).cuda(),
        "subcells": torch.from_numpy(subcells).cuda(), "x0": x0, "v0": v0, "magnetic": magnetic,
        "active": torch.arange(n, **ints), "x": torch.empty_like(x0), "v": torch.empty_like(v0),
        "qm": torch.full((n,), CHARGE / PROTON, **f64), "dq": torch.full((n,), 1e-3 / n, **f64),
        "steps": torch.zeros(n, **ints), "status": torch.zeros(n, **ints),
        "electrode": torch.zeros(n, **ints), "inside": inside,
        "patch_int": torch.tensor([[*mesh.shape, 0, 0, 0, nodes, 0]], **ints),
        "patch_real": torch.tensor([[*mesh.origin, mesh.h, *mesh.origin, *mesh.upper]], **f64),
        "planes": torch.tensor([20.0 * MM, 79.0 * MM], **f64),
        "hits": torch.zeros((n, 2, 4, 8), **f64), "counts": torch.zeros((n, 2), **ints),
        "path_slot": torch.full((n,), -1, **ints), "paths": torch.zeros((1, 1, 3), **f64),
        "path_count": torch.ones(1, **ints), "charge": torch.zeros((1, nodes), **f64),
        "current": torch.zeros((1, 3 * nodes if case["current"] else 1), **f64),
        "integrator": case["integrator"], "has_b": int(case["magnetic"]),
        "has_j": int(case["current"]),
    }  # fmt: skip


# -- one pass -------------------------------------------------------------------------------------


def run(state: dict):
    kind = state["kind"]
    if kind == "gather":
        KERNELS["staggered_field_2d"](state["px"], state["py"], state["fx"], state["fy"], 0.0, 0.0,
                                      state["h"], state["ex"], state["ey"])  # fmt: skip
        return {"ex": state["ex"], "ey": state["ey"]}
    if kind == "deposit":
        state["charge"].zero_()
        KERNELS["deposit_trajectories_2d"](state["px"], state["py"], state["q"], 0.0, 0.0,
                                           state["h"], int(state["cylindrical"]), state["charge"])  # fmt: skip
        return {"charge": state["charge"]}
    if kind == "field":
        state["phi"].zero_()
        state["solver"].solve_device(state["phi"], state["rho"])
        return {"phi": state["phi"]}
    if kind in ("plasma", "refined"):
        state["phi"].copy_(state["first"])
        state["solver"].solve_device(state["phi"], state["rho"], plasma=state["species"])
        return {"phi": state["phi"]}
    if kind in ("trace", "magnetic"):
        engine = state["engine"]
        engine.run(state["fx"], state["fy"])
        return {"x": engine.x, "v": engine.v, "steps": engine.steps, "status": engine.status,
                "electrode": engine.electrode, "hits": engine.hits, "counts": engine.counts,
                "charge": engine.charge}  # fmt: skip
    if kind == "trace3d":
        return _run_3d(state)
    if kind == "adjoint":
        state["adjoint"].record()
        fx_bar, fy_bar = state["adjoint"].sweep(state["charge_seed"], state["hit_seed"])
        return {"fx_bar": fx_bar, "fy_bar": fy_bar}
    if kind in ("diode", "lens"):
        model = BeamOptics(state["config"]).run()
        out = {"potential": model.potential, "charge_density": model.charge_density,
               "status": model.state.trace.status}  # fmt: skip
        for k, x in enumerate(state["config"].diagnostic_planes):
            moments = model.beam_moments(x)
            out[f"moments{k}"] = np.array([moments.current, moments.rms_size, moments.rms_angle,
                                           moments.emittance])  # fmt: skip
        return out
    batch = BatchedVlasov(state["configs"]).run()
    moments = [c.moments(79 * MM) for c in batch.candidates]
    batch.close()
    return {"phi": batch.phi, "rho": batch.rho, "status": batch.status,
            "moments": np.array([[m.current, m.rms_size, m.rms_angle] for m in moments])}  # fmt: skip


def _run_3d(s: dict) -> dict:
    s["x"].copy_(s["x0"])
    s["v"].copy_(s["v0"])
    s["status"].fill_(-1)
    s["electrode"].fill_(-1)
    for name in ("steps", "counts", "charge", "current"):
        s[name].zero_()
    mesh, e = s["mesh"], s["electric"]
    KERNELS["trace_trajectories_3d"](
        s["active"], s["x"], s["v"], s["qm"], s["dq"], s["steps"], s["status"], s["electrode"],
        e.fx_device, e.fy_device, e.fz_device, s["patch_int"], s["patch_real"], s["magnetic"],
        s["has_b"], *mesh.origin, mesh.h, *mesh.upper, 0, 0, s["integrator"], 0.5, 100_000,
        s["cells"], s["subcells"], 4, s["planes"], s["hits"], s["counts"], s["path_slot"],
        s["paths"], s["path_count"], 1, s["charge"], s["has_j"], s["current"], 0.0)  # fmt: skip
    names = ("x", "v", "steps", "status", "electrode", "hits", "counts", "charge", "current")
    return {name: s[name] for name in names}


# -- what a pass cannot do without ----------------------------------------------------------------

#: Operations of one Runge-Kutta step of a 2D trace, its gathers and deposit included.
STEP_FLOPS = 370


def _trace_work(nodes: int, n: int, steps: float, flops: float) -> dict:
    # the beam's states, charges and masses in, its ends and crossings out; the edge fields
    # in and the node charges out
    return {"bytes": n * (8 * 8 + 9 * 8 + 2 * 64) + nodes * 24, "flops": n * steps * flops}


def work(case: dict) -> dict:
    kind = case["kind"]
    ny = case.get("ny", 0)
    nx = case.get("nx", 4 * (ny - 1) + 1)
    nodes = nx * ny
    if kind == "gather":
        return {"bytes": 32 * case["points"] + 16 * nodes, "flops": 30 * case["points"]}
    if kind == "deposit":
        return {"bytes": 24 * case["points"] + 8 * nodes, "flops": 20 * case["points"]}
    # a field solve reads its density and rows and writes the potential; its operations are
    # those of a dozen multigrid cycles of two sweeps before and after the correction
    field = {"bytes": 64 * nodes, "flops": 12 * 4 * 13 * nodes}
    if kind == "field":
        return field
    if kind == "plasma":
        return {"bytes": field["bytes"], "flops": 4 * field["flops"]}
    if kind == "refined":
        count = nodes * (1 + case["boxes"]) * (4 if case["plasma"] else 1)
        return {"bytes": 64 * nodes * (1 + case["boxes"]), "flops": 12 * 4 * 13 * count}
    if kind in ("trace", "adjoint"):
        flops = {"rk4": STEP_FLOPS, "boris": 190}[case.get("integrator", "rk4")]
        return _trace_work(nodes, case["rings"], 2 * nx, flops * (4 if kind == "adjoint" else 1))
    if kind == "magnetic":
        return _trace_work(nodes, case["trajectories"], 4 * ny, 260)
    if kind == "trace3d":
        m = case["cells"]
        per_step = (600 if case["integrator"] == 0 else 320) + (200 if case["magnetic"] else 0)
        return _trace_work(4 * m**3, case["trajectories"], 8 * m, per_step)
    if kind in ("diode", "lens"):
        n = case.get("rings", case.get("trajectories"))
        trace = _trace_work(nodes, n, 2 * nx, STEP_FLOPS)
        return {"bytes": 6 * (field["bytes"] + trace["bytes"]),
                "flops": 6 * (field["flops"] + trace["flops"])}  # fmt: skip
    count = case["candidates"]
    nodes, n = 100_000 * count, 11_000 * count
    trace = _trace_work(nodes, n, 1_200, STEP_FLOPS)
    return {"bytes": 8 * (64 * nodes + trace["bytes"]),
            "flops": 8 * (12 * 4 * 13 * nodes + trace["flops"])}  # fmt: skip


# -- the outputs from plain torch in 64 bits -----------------------------------------------------


def _bilinear(f, s, t):
    """``f`` at fractional indices, the cell clamped to the array."""
    i = torch.floor(s).long().clamp(0, f.shape[0] - 2)
    j = torch.floor(t).long().clamp(0, f.shape[1] - 2)
    u, w = s - i, t - j
    low = f[i, j] + w * (f[i, j + 1] - f[i, j])
    high = f[i + 1, j] + w * (f[i + 1, j + 1] - f[i + 1, j])
    return low + u * (high - low)


def _trilinear(f, s, t, u):
    i = torch.floor(s).long().clamp(0, f.shape[0] - 2)
    j = torch.floor(t).long().clamp(0, f.shape[1] - 2)
    k = torch.floor(u).long().clamp(0, f.shape[2] - 2)
    a, b, c = s - i, t - j, u - k
    out = 0.0
    for di, wi in ((0, 1.0 - a), (1, a)):
        for dj, wj in ((0, 1.0 - b), (1, b)):
            for dk, wk in ((0, 1.0 - c), (1, c)):
                out = out + wi * wj * wk * f[i + di, j + dj, k + dk]
    return out


def _cell(s, n):
    """The cell of fractional indices along an axis of n nodes and the weight in it, both
    clamped to the axis."""
    i = torch.floor(s).long()
    w = (s - i).where((i >= 0) & (i < n - 1), (i >= n - 1).double())
    return i.clamp(0, n - 2), w


def _add_2d(charge, sx, r, q, h, y0, cylindrical):
    """Area-weighted charges added to the nodes (the areas of rings when cylindrical)."""
    nx, ny = charge.shape
    i, u = _cell(sx, nx)
    sy = (r - y0) / h
    j, w = _cell(sy, ny)
    if cylindrical:
        low = y0 + h * j.double()
        ring = (r * r - low * low) / ((low + h) ** 2 - low * low)
        w = ring.where((sy >= 0) & (sy < ny - 1), w)
    flat = charge.view(-1)
    for di, a in ((0, 1.0 - u), (1, u)):
        for dj, b in ((0, 1.0 - w), (1, w)):
            flat.index_add_(0, (i + di) * ny + j + dj, a * b * q)


def _rows(mesh, fixed):
    """The field's neighbour coefficients (west, east, south, north) on the free nodes."""
    nx, ny = mesh.shape
    f64 = dict(dtype=torch.float64, device="cuda")
    x = torch.from_numpy(np.array(mesh.x)).cuda()
    a, b, c, d = torch.from_numpy(np.array(mesh.distance)).cuda()
    h, hx = float(mesh.h), (x[1:] - x[:-1])[:, None]
    west, east, south, north = (torch.zeros((nx, ny), **f64) for _ in range(4))
    inside = torch.zeros((nx, ny), dtype=torch.bool, device="cuda")
    inside[1:-1, 1:-1] = True

    def pair(low, high, control):
        # Shortley and Weller's row where all four cells exist, else the edges' fluxes
        return (torch.where(control > 0, 1.0 / (control * low), 2.0 / ((low + high) * low)),
                torch.where(control > 0, 1.0 / (control * high), 2.0 / ((low + high) * high)))  # fmt: skip

    control = torch.where(inside, 0.0, 1.0)[1:-1] * 0.5 * (hx[:-1] + hx[1:])
    west[1:-1], east[1:-1] = pair(a[1:-1] * hx[:-1], b[1:-1] * hx[1:], control)
    east[0], west[-1] = 2.0 / (hx[0] * hx[0] * b[0]), 2.0 / (hx[-1] * hx[-1] * a[-1])
    if not mesh.cylindrical:
        control = torch.where(inside, 0.0, h)[:, 1:-1]
        south[:, 1:-1], north[:, 1:-1] = pair(c[:, 1:-1] * h, d[:, 1:-1] * h, control)
        north[:, 0] = 2.0 / (h * h * d[:, 0])
    else:
        k = torch.arange(ny, **f64)[None, 1:-1]
        p, q, four = c[:, 1:-1], d[:, 1:-1], inside[:, 1:-1]
        south[:, 1:-1] = torch.where(four, (2.0 / p - 1.0 / k) / (p + q), (1.0 - 0.5 / k) / p) / h**2
        north[:, 1:-1] = torch.where(four, (2.0 / q + 1.0 / k) / (p + q), (1.0 + 0.5 / k) / q) / h**2
        north[:, 0] = 4.0 / (h * h * d[:, 0])
    south[:, -1] = 2.0 / (h * h * c[:, -1])
    return [torch.where(fixed, 0.0, m) for m in (west, east, south, north)]


def _solve(rows, fixed, right, extra=None):
    """The potential of the rows: block elimination along x, a column of nodes a block."""
    west, east, south, north = rows
    nx, ny = right.shape
    diagonal = west + east + south + north + fixed.double()
    if extra is not None:
        diagonal = diagonal + extra
    eye = torch.eye(ny, dtype=torch.float64, device=right.device)
    coupling, load = [], []
    for i in range(nx):
        block = torch.diag(diagonal[i]) - torch.diag(south[i, 1:], -1) - torch.diag(north[i, :-1], 1)
        b = right[i]
        if i:
            block = block - west[i][:, None] * coupling[-1]
            b = b + west[i] * load[-1]
        solved = torch.linalg.solve(block, torch.cat([eye * east[i], b[:, None]], dim=1))
        coupling.append(solved[:, :ny])
        load.append(solved[:, ny])
    phi = torch.empty_like(right)
    phi[-1] = load[-1]
    for i in range(nx - 2, -1, -1):
        phi[i] = load[i] + coupling[i] @ phi[i + 1]
    return phi


def _field(mesh, rho, species=None):
    fixed = torch.from_numpy(np.array(mesh.fixed)).cuda()
    value = torch.from_numpy(np.array(mesh.fixed_value)).cuda()
    rows = _rows(mesh, fixed)
    right = torch.where(fixed, value, rho / EPS0)
    if species is None:
        return _solve(rows, fixed, right)
    amplitude, t, up = species.rho_e / EPS0, species.electron_temperature, species.plasma_potential
    phi = species.first
    phi = torch.where(fixed, value, phi)
    for _ in range(40):
        e = torch.where(fixed, 0.0, amplitude * torch.exp(((phi - up) / t).clamp(max=50.0)))
        # Newton's step as the next potential: (A + e / T) phi' = b - e + e phi / T
        new = _solve(rows, fixed, right - e + e * phi / t, e / t)
        change = float((new - phi).abs().max())
        phi = new
        if change < 1e-7:
            break
    return phi


def _integrate(fields, spacing, boris, qm, dq, x, v, ended, add, cross, most=100_000):
    """Trajectories to their ends: ``fields(q) -> (E, B)``; ``spacing(x)`` the local cell;
    ``ended(x)`` where a step's end finishes a trajectory; ``add`` takes a step's midpoint
    and charge, ``cross`` its two ends.  Returns the last positions and velocities."""
    x, v = x.clone(), v.clone()
    out_x, out_v = x.clone(), v.clone()
    at = torch.arange(x.shape[1], device=x.device)
    norm = lambda a: torch.sqrt((a * a).sum(0))  # noqa: E731
    turn = lambda a, b: torch.stack([a[1] * b[2] - a[2] * b[1], a[2] * b[0] - a[0] * b[2],  # noqa: E731
                                     a[0] * b[1] - a[1] * b[0]])  # fmt: skip

    def pull(q, u, qm):
        e, b = fields(q)
        return qm * (e if b is None else e + turn(u, b))

    def kick(u, q, tau, qm):
        e, b = fields(q)
        f = 0.5 * tau * qm
        if b is None:
            return u + 2.0 * f * e
        m, t = u + f * e, f * b
        s = 2.0 * t / (1.0 + (t * t).sum(0))
        return m + turn(m + turn(m, t), s) + f * e

    for count in range(1, most + 1):
        m, c = qm[at], dq[at]
        a = pull(x, v, m)
        h = spacing(x)
        dt = 0.5 * torch.minimum(h / norm(v), torch.sqrt(2.0 * h / norm(a)))
        half = 0.5 * dt
        if boris:
            w = kick(v, x, half, m)
            y = x + dt * w
            w = kick(w, y, half, m)
        else:
            k1 = v + half * a
            a1 = pull(x + half * v, k1, m)
            k2 = v + half * a1
            a2 = pull(x + half * k1, k2, m)
            k3 = v + dt * a2
            a3 = pull(x + dt * k2, k3, m)
            y = x + dt / 6.0 * (v + 2.0 * k1 + 2.0 * k2 + k3)
            w = v + dt / 6.0 * (a + 2.0 * a1 + 2.0 * a2 + a3)
        add(0.5 * (x + y) + dt * (v - w) * 0.125, c * dt, c * (y - x))
        cross(at, count, x, v, y, w)
        x, v = y, w
        done = ended(x)
        if bool(done.any()):
            out_x[:, at[done]], out_v[:, at[done]] = x[:, done], v[:, done]
            x, v, at = x[:, ~done], v[:, ~done], at[~done]
            if not at.numel():
                break
    return out_x, out_v


def _crossings(n, planes, capacity=4):
    hits = torch.zeros((n, len(planes), capacity, 8), dtype=torch.float64, device="cuda")
    counts = torch.zeros((n, len(planes)), dtype=torch.int64, device="cuda")

    def cross(at, step, x, v, y, w):
        for p, position in enumerate(planes):
            before, after = x[0] - position, y[0] - position
            i = torch.nonzero((before < 0) != (after < 0)).flatten()
            if not i.numel():
                continue
            t = before[i] / (before[i] - after[i])
            k = at[i]
            record = torch.stack([
                torch.full_like(t, position), *(x[1:, i] + t * (y[1:, i] - x[1:, i])),
                *(v[:, i] + t * (w[:, i] - v[:, i])),
                torch.where(after[i] >= 0, 1.0, -1.0), torch.full_like(t, float(step))], dim=1)  # fmt: skip
            c = counts[k, p]
            held = c < capacity
            hits[k[held], p, c[held]] = record[held]
            counts[k, p] += 1

    return hits, cross


def _trace_2d(mesh, fx, fy, particles, planes, boris, inside, magnetic=None):
    """The trace of a beam on a 2D mesh: ends, crossings and node charges."""
    nx, ny = mesh.shape
    cylindrical, h = mesh.cylindrical, float(mesh.h)
    x0, y0 = mesh.origin
    (_, top), nodes = mesh.upper, torch.from_numpy(np.array(mesh.x)).cuda()
    right = float(nodes[-1])
    fx, fy = fx.view(nx + 1, ny), fy.view(nx, ny + 1)
    put = lambda a: torch.from_numpy(np.array(a, dtype=np.float64)).cuda()  # noqa: E731
    charge = torch.zeros((nx, ny), dtype=torch.float64, device="cuda")

    def fraction(x):  # the fractional node index along x
        if not mesh.graded:
            return (x - x0) / h
        i = torch.searchsorted(nodes, x.contiguous(), right=True).sub(1).clamp(0, nx - 2)
        return i + (x - nodes[i]) / (nodes[i + 1] - nodes[i])

    def across(q):  # the mesh's second coordinate
        return torch.sqrt(q[1] * q[1] + q[2] * q[2]) if cylindrical else q[1]

    def fields(q):
        r = across(q)
        sx, sy = fraction(q[0]), (r - y0) / h
        ex, ey = _bilinear(fx, sx + 0.5, sy), _bilinear(fy, sx, sy + 0.5)
        if cylindrical:
            unit = torch.where(r > 0, 1.0 / r, 0.0)
            e = torch.stack([ex, ey * q[1] * unit, ey * q[2] * unit])
        else:
            e = torch.stack([ex, ey, torch.zeros_like(ex)])
        return e, None if magnetic is None else magnetic(q)

    def spacing(x):
        if not mesh.graded:
            return torch.full_like(x[0], h)
        i = torch.floor(fraction(x[0])).long().clamp(0, nx - 2)
        return torch.minimum(nodes[i + 1] - nodes[i], torch.full_like(x[0], h))

    def ended(x):
        r = across(x)
        out = (x[0] >= right) | (x[0] < x0) | (r > top) | inside(x[0], r)
        return out if cylindrical else out | (r < y0)

    def add(middle, q, _):
        _add_2d(charge, fraction(middle[0]), across(middle), q, h, y0, cylindrical)

    n = len(particles)
    hits, cross = _crossings(n, planes or (math.nan,))
    x, v = _integrate(fields, spacing, boris, put(particles.charge / particles.mass),
                      put(np.sign(particles.charge) * np.abs(particles.current)),
                      put(particles.position), put(particles.velocity), ended, add, cross)  # fmt: skip
    return {"x": x, "v": v, "steps": None, "status": None, "electrode": None, "hits": hits,
            "counts": None, "charge": charge.view(1, -1)}  # fmt: skip


def _exact_trace(case: dict, seed: int):
    state = prepare(case, seed)
    mesh, particles = state["mesh"], state["engine"].particles
    if case["kind"] == "trace":
        design = _lens_design(case, seed)

        def inside(x, r):
            hit = torch.zeros_like(x, dtype=torch.bool)
            for centre in design.centres:
                hit |= ((x - centre).abs() <= 0.5 * design.thickness) & (r >= design.aperture)
            return hit

        return _trace_2d(mesh, state["fx"], state["fy"], particles, design.planes,
                         case["integrator"] == "boris", inside)  # fmt: skip
    design, field = state["design"], state["field"]
    bz = torch.from_numpy(np.array(field.bz)).cuda()
    slope = torch.zeros_like(bz)
    # the sixth-order central difference of the on-axis samples
    weights = (-1 / 60, 9 / 60, -45 / 60, 0.0, 45 / 60, -9 / 60, 1 / 60)
    for k, weight in enumerate(weights):
        slope[3:-3] += weight * bz[k : bz.numel() - 6 + k] / field.hz

    def magnetic(q):
        s = (q[0] - field.z0) / field.hz
        i = torch.floor(s).long().clamp(3, bz.numel() - 5)
        t = s - i
        along = bz[i] + t * (bz[i + 1] - bz[i])
        change = slope[i] + t * (slope[i + 1] - slope[i])
        return torch.stack([along, -0.5 * (q[1] - design.axis_y) * change, torch.zeros_like(along)])

    def inside(x, y):
        hit = torch.zeros_like(x, dtype=torch.bool)
        for low, high in (design.plasma_electrode, design.extraction_electrode):
            hit |= (x >= low) & (x <= high) & ((y - design.axis_y).abs() >= 0.5 * design.slit)
        return hit

    return _trace_2d(mesh, state["fx"], state["fy"], particles, (), True, inside, magnetic)


def _exact_3d(case: dict, seed: int):
    s = prepare(case, seed)
    mesh, e = s["mesh"], s["electric"]
    h, shape = float(mesh.h), mesh.shape
    upper = torch.tensor(mesh.upper, dtype=torch.float64, device="cuda")[:, None]
    charge = torch.zeros(shape, dtype=torch.float64, device="cuda")
    current = torch.zeros((3, *shape), dtype=torch.float64, device="cuda")
    cells, subcells = s["cells"], s["subcells"].view(-1, 4, 4, 4)

    def fields(q):
        a, b, c = q / h
        ef = torch.stack([_trilinear(e.fx_device, a + 0.5, b, c), _trilinear(e.fy_device, a, b + 0.5, c),
                          _trilinear(e.fz_device, a, b, c + 0.5)])  # fmt: skip
        if not case["magnetic"]:
            return ef, None
        return ef, torch.stack([_trilinear(m, a, b, c) for m in s["magnetic"]])

    def ended(x):
        off = (x >= upper)[0] | (x > upper).any(0) | (x < 0).any(0)
        # in an electrode's sub-cell, or in one its surface cuts (the caller's to decide)
        u = x / h
        limit = torch.tensor([n - 2 for n in shape], device="cuda")[:, None]
        i = torch.minimum(u.long().clamp(min=0), limit)
        number = cells[i[0], i[1], i[2]]
        j = ((u - i) * 4).long().clamp(0, 3)
        sub = subcells[number.clamp(min=0), j[0], j[1], j[2]]
        return off | ((number >= 0) & (sub != -1))

    def add(middle, q, moved):
        (i, a), (j, b), (k, c) = (_cell(middle[d] / h, shape[d]) for d in range(3))
        for di, wi in ((0, 1.0 - a), (1, a)):
            for dj, wj in ((0, 1.0 - b), (1, b)):
                for dk, wk in ((0, 1.0 - c), (1, c)):
                    at = ((i + di) * shape[1] + j + dj) * shape[2] + k + dk
                    charge.view(-1).index_add_(0, at, wi * wj * wk * q)
                    if case["current"]:
                        for d in range(3):
                            current[d].view(-1).index_add_(0, at, wi * wj * wk * moved[d])

    hits, cross = _crossings(case["trajectories"], s["planes"].tolist())
    x, v = _integrate(fields, lambda x: torch.full_like(x[0], h), case["integrator"] == 1, s["qm"],
                      s["dq"], s["x0"], s["v0"], ended, add, cross)  # fmt: skip
    return {"x": x, "v": v, "steps": None, "status": None, "electrode": None, "hits": hits,
            "counts": None, "charge": charge.view(1, -1),
            "current": current.view(1, -1) if case["current"] else s["current"]}  # fmt: skip


def _exact_diode(case: dict, seed: int):
    """The diode's iterations: the field, its edges, the trace, the density."""
    config = _diode_config(case, seed)
    mesh = BeamOptics(config).mesh
    particles, _ = config_particles(config)
    nx, ny = mesh.shape
    h = float(mesh.h)
    rho = torch.zeros((nx, ny), dtype=torch.float64, device="cuda")
    volumes = torch.full((nx, ny), h * h, dtype=torch.float64, device="cuda")
    for face in (volumes[0], volumes[-1], volumes[:, 0], volumes[:, -1]):
        face *= 0.5
    nowhere = lambda x, y: torch.zeros_like(x, dtype=torch.bool)  # noqa: E731
    previous = None
    for _ in range(config.iterations):
        phi = _field(mesh, rho)
        # the field on the edges between nodes, extended linearly past the faces
        ex, ey = (phi[:-1] - phi[1:]) / h, (phi[:, :-1] - phi[:, 1:]) / h
        fx = torch.cat([2.0 * ex[:1] - ex[1:2], ex, 2.0 * ex[-1:] - ex[-2:-1]])
        fy = torch.cat([2.0 * ey[:, :1] - ey[:, 1:2], ey, 2.0 * ey[:, -1:] - ey[:, -2:-1]], dim=1)
        out = _trace_2d(mesh, fx.contiguous(), fy.contiguous(), particles,
                        config.diagnostic_planes, False, nowhere)  # fmt: skip
        rho = out["charge"].view(nx, ny) / volumes
        if previous is not None and float((phi - previous).abs().max()) < config.tolerance:
            break
        previous = phi
    return {"potential": phi, "charge_density": rho, "status": None, "moments0": None}


class _Species:
    """A Boltzmann species with the first guess its Newton iteration starts from."""

    def __init__(self, species, first) -> None:
        self.rho_e, self.plasma_potential = species.rho_e, species.plasma_potential
        self.electron_temperature, self.first = species.electron_temperature, first


def exact(case: dict, seed: int):
    kind = case["kind"]
    if kind == "gather":
        s = prepare(case, seed)
        a, b = s["px"] / s["h"], s["py"] / s["h"]
        return {"ex": _bilinear(s["fx"], a + 0.5, b), "ey": _bilinear(s["fy"], a, b + 0.5)}
    if kind == "deposit":
        s = prepare(case, seed)
        charge = torch.zeros_like(s["charge"])
        _add_2d(charge, s["px"] / s["h"], s["py"], s["q"], s["h"], 0.0, case["cylindrical"])
        return {"charge": charge}
    if kind == "field":
        s = prepare(case, seed)
        return {"phi": _field(s["mesh"], s["rho"])}
    if kind == "plasma":
        # a direct elimination for each of some ten Newton steps: minutes on a large mesh
        if case["nx"] * case["ny"] ** 1.5 > 1.5e6:
            return None
        s = prepare(case, seed)
        return {"phi": _field(s["mesh"], s["rho"], _Species(s["species"], s["first"]))}
    if kind in ("trace", "magnetic"):
        return _exact_trace(case, seed)
    if kind == "trace3d":
        return _exact_3d(case, seed)
    if kind == "diode":
        return _exact_diode(case, seed)
    # refined boxes, reverse sweeps and whole converged solves: minutes in plain torch
    return None
