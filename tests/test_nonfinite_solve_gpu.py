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


@pytest.mark.parametrize("value", [np.nan, np.inf])
def test_a_batch_refuses_a_nonfinite_candidate(value):
    """The candidate's own solves are refused; the batch then solves finite densities."""
    from beamtracer_b200._lib import ConvergenceError
    from tests.test_batch_gpu import DESIGNS, _batch

    batch = _batch(DESIGNS[:2])
    batch.node_view(batch.rho, 1)[80, 5] = value
    with pytest.raises(ConvergenceError):
        batch.poisson_batch.solve(batch.phi, batch.rho, [0, 1])
    batch.rho.zero_()
    batch.phi.zero_()
    batch.poisson_batch.solve(batch.phi, batch.rho, [0, 1])
    assert bool(batch.phi.isfinite().all())
