"""The coarsest level's inverse: meshes small enough to be their own coarsest level."""

from __future__ import annotations

import numpy as np
import pytest

from beamtracer_b200.mesh import Electrode, FaceCondition, IonOpticsMesh
from oracle import poisson as oracle

pytestmark = pytest.mark.gpu

# half-bandwidths 4 to 17 (the shorter side plus one, either axis), at the edges of the
# substitution's widths (6, 10, 14, 18) and of its 32-column blocks, and the largest level
SHAPES = [(3, 3), (3, 85), (85, 3), (5, 6), (6, 42), (9, 28), (28, 9), (10, 25), (13, 19),
          (14, 18), (16, 16), (15, 17), (8, 8), (11, 3)]  # fmt: skip


@pytest.mark.parametrize("geometry", ["planar", "cylindrical"])
@pytest.mark.parametrize("shape", SHAPES, ids=str)
def test_coarsest_inverse(shape, geometry):
    """The dense inverse solves the mesh's own operator: the first V-cycle reaches the
    rounding floor (1e-16 times the operator's condition, below 1e5 here), so three cycles
    meet a residual of 1e-13, and the potential is the oracle's LU to 1e-9 of its span."""
    from beamtracer_b200.poisson import IonOpticsPoisson

    h = 1e-3
    faces = {"x_min": FaceCondition("dirichlet", 0.0), "x_max": FaceCondition("dirichlet", 100.0)}
    far = (shape[0] - 1) * h
    rod = Electrode(lambda x, y: (np.abs(x - 0.5 * far) <= 0.3 * far) & (y >= (shape[1] - 1.4) * h),
                    -40.0)  # fmt: skip
    mesh = IonOpticsMesh(shape=shape, origin=(0.0, 0.0), h=h, geometry=geometry,
                         electrodes=[rod], faces=faces)  # fmt: skip
    rho = np.random.default_rng(4).uniform(0.0, 1e-5, shape)
    solver = IonOpticsPoisson(mesh)
    phi = solver.solve(rho)
    expected = oracle.solve(oracle.operator_of_mesh(mesh), rho)
    assert solver.krylov_steps <= 3
    np.testing.assert_allclose(phi, expected, rtol=0, atol=1e-9 * max(np.ptp(expected), 1.0))
