"""The reverse sweep of trajectories that took no step, among others in their warp."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("steps", [0, -1, -128, -1000])
def test_trajectories_of_no_step_add_nothing(steps):
    """A trajectory whose step count is zero or negative is left out: the sweep is that of the
    others, to the rounding of some 1e3 additions per edge (1e-11 of the largest)."""
    import torch

    from beamtracer_b200.adjoint import TraceAdjoint
    from beamtracer_b200.einzel import EinzelDesign, einzel_config
    from beamtracer_b200.fields import StaggeredElectricField
    from beamtracer_b200.model import BeamOptics, config_particles
    from beamtracer_b200.poisson import IonOpticsPoisson
    from beamtracer_b200.tracer import TraceEngine

    count = 40
    config = einzel_config(EinzelDesign(shape=(161, 41), trajectories=count, seed=4,
                                        voltages=(0.0, 8e3, 0.0)))  # fmt: skip
    mesh = BeamOptics(config).mesh
    phi = torch.zeros(mesh.shape, dtype=torch.float64, device="cuda")
    IonOpticsPoisson(mesh).solve_device(phi)
    field = StaggeredElectricField(mesh, phi)
    particles, _ = config_particles(config)
    charge_seed = torch.from_numpy(np.random.default_rng(1).normal(size=mesh.shape)).cuda()

    def sweep(beam, without=()):
        engine = TraceEngine(mesh, planes=(70e-3, 79e-3))
        engine.load(beam)
        engine.run(field.fx_device, field.fy_device)
        for k in without:
            engine.steps[k] = steps
        adjoint = TraceAdjoint(engine, field.fx_device, field.fy_device)
        adjoint.record()
        seed = torch.ones_like(engine.hits) * 1e-3
        return torch.cat([b.reshape(-1) for b in adjoint.sweep(charge_seed, seed)])

    without = (3, 17, 35)
    kept = np.setdiff1d(np.arange(count), without)
    expected = sweep(particles.subset(kept))
    assert float(expected.abs().max()) > 0.0
    got = sweep(particles, without)
    assert float((got - expected).abs().max()) <= 1e-11 * float(expected.abs().max())
