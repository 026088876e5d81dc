"""A residual that is no number, or infinite, must not read as a converged field."""

from __future__ import annotations

import numpy as np
import pytest

from tests.test_poisson_gpu import _plates

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("plasma", [False, True])
@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf])
@pytest.mark.parametrize("where", ["rho", "phi"])
def test_nonfinite_input_is_refused(where, value, plasma):
    """One such value on a free node, in the charge density or the first guess; the same solver
    then solves a finite problem as a new one does."""
    import torch

    from beamtracer_b200._lib import ConvergenceError
    from beamtracer_b200.poisson import BoltzmannElectrons, IonOpticsPoisson

    species = BoltzmannElectrons(1e-6, 5.0, 50.0) if plasma else None
    solver = IonOpticsPoisson(_plates((33, 17)))
    arrays = {k: torch.zeros((33, 17), dtype=torch.float64, device="cuda") for k in ("rho", "phi")}
    arrays[where][16, 8] = value
    with pytest.raises(ConvergenceError):
        solver.solve_device(arrays["phi"], arrays["rho"], plasma=species)
    expected = IonOpticsPoisson(_plates((33, 17))).solve(plasma=species)
    assert np.array_equal(solver.solve(plasma=species), expected)
