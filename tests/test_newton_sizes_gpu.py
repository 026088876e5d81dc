"""The hierarchy of ragged meshes and Newton's updates on them, against the oracle."""

from __future__ import annotations

import numpy as np
import pytest
from scipy.constants import epsilon_0

from beamtracer_b200.mesh import Electrode, FaceCondition, IonOpticsMesh
from oracle import poisson as oracle

pytestmark = pytest.mark.gpu

# odd and even sides (an even side's last coarse cell is one fine cell), a side too short to
# coarsen, node counts below, at and past a block of fine and of coarse nodes
SHAPES = [(17, 33), (34, 18), (3, 130), (65, 20), (97, 101), (130, 67)]


@pytest.mark.parametrize("geometry", ["planar", "cylindrical"])
@pytest.mark.parametrize("shape", SHAPES, ids=str)
def test_newton_on_ragged_meshes(shape, geometry):
    """The linear solve within one Krylov cycle (30 V-cycles: a hierarchy that contracts the
    residual by 0.35 a cycle needs 29 for 1e-13) and Newton's potential, both to 1e-9 of the
    span of the oracle's LU."""
    from beamtracer_b200.poisson import BoltzmannElectrons, IonOpticsPoisson

    h = 0.2e-3
    far, top = (shape[0] - 1) * h, (shape[1] - 1) * h
    faces = {"x_min": FaceCondition("dirichlet", 10.0), "x_max": FaceCondition("dirichlet", -200.0)}
    plate = Electrode(lambda x, y: (np.abs(x - 0.4 * far) <= 0.1 * far) & (y >= 0.6 * top), -30.0)
    mesh = IonOpticsMesh(shape=shape, origin=(0.0, 0.0), h=h, geometry=geometry,
                         electrodes=[plate], faces=faces)  # fmt: skip
    rho = np.random.default_rng(1).uniform(0.0, 1e-4, shape)
    operator = oracle.operator_of_mesh(mesh)
    solver = IonOpticsPoisson(mesh)
    linear = solver.solve(rho)
    expected = oracle.solve(operator, rho)
    assert solver.krylov_steps <= 30
    span = np.ptp(expected)
    np.testing.assert_allclose(linear, expected, rtol=0, atol=1e-9 * span)
    density = 5e-5
    phi = solver.solve(rho, plasma=BoltzmannElectrons(density, 5.0, 10.0), tolerance=1e-12)
    expected, _ = oracle.solve_newton(operator, rho, density / epsilon_0, 5.0, 10.0, -1, tol=1e-10)
    np.testing.assert_allclose(phi, expected, rtol=0, atol=1e-9 * span)
