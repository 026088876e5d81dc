"""The reverse sweep of trajectories of very different lengths in one warp."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("count", [1, 31, 33, 70])
def test_the_sweep_of_a_beam_is_the_sum_of_its_trajectories(count):
    """The edge fields' adjoint is a sum over trajectories: swept together -- lengths from a
    few steps to several segments of 64 in one warp, one on the axis, a last warp not full --
    it equals the trajectories swept alone, summed, to the rounding of some 1e3 additions per
    edge (1e-11 of the largest)."""
    import torch

    from beamtracer_b200.adjoint import TraceAdjoint
    from beamtracer_b200.einzel import EinzelDesign, einzel_config
    from beamtracer_b200.fields import StaggeredElectricField
    from beamtracer_b200.model import BeamOptics, config_particles
    from beamtracer_b200.poisson import IonOpticsPoisson
    from beamtracer_b200.tracer import TraceEngine

    config = einzel_config(EinzelDesign(shape=(161, 41), trajectories=count, seed=4,
                                        voltages=(0.0, 8e3, 0.0)))  # fmt: skip
    mesh = BeamOptics(config).mesh
    phi = torch.zeros(mesh.shape, dtype=torch.float64, device="cuda")
    IonOpticsPoisson(mesh).solve_device(phi)
    field = StaggeredElectricField(mesh, phi)
    particles, _ = config_particles(config)
    particles.position[0] = np.linspace(1e-3, 78e-3, count) if count > 1 else 1e-3
    particles.position[1:, 0] = 0.0  # on the axis, along it
    particles.velocity[1:, 0] = 0.0
    rng = np.random.default_rng(count)
    charge_seed = torch.from_numpy(rng.normal(size=mesh.shape)).cuda()

    def sweep(beam, hits=None):
        engine = TraceEngine(mesh, planes=(70e-3, 79e-3))
        engine.load(beam)
        engine.run(field.fx_device, field.fy_device)
        adjoint = TraceAdjoint(engine, field.fx_device, field.fy_device)
        adjoint.record()
        seed = torch.ones_like(engine.hits) * 1e-3
        return torch.cat([b.reshape(-1) for b in adjoint.sweep(charge_seed, seed)]), engine.steps

    together, steps = sweep(particles)
    if count > 1:
        assert int(steps.min()) < 64 < 256 < int(steps.max())
    alone = sum(sweep(particles.subset(slice(k, k + 1)))[0] for k in range(count))
    assert float(alone.abs().max()) > 0.0
    assert float((together - alone).abs().max()) <= 1e-11 * float(alone.abs().max())
