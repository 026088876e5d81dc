"""A V-cycle whose result overlaps its right-hand side (``bt_poisson_vcycle``)."""

from __future__ import annotations

import numpy as np
import pytest

from tests.test_poisson_gpu import _plates, _three_plates

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("staged", [True, False])
@pytest.mark.parametrize("shape", [(15, 17), (41, 21), (257, 65)], ids=str)
def test_overlapping_vcycle(shape, staged):
    """In place, or shifted by part of the vector either way, the cycle gives the bits it
    gives with vectors apart: on a mesh of one level, of a tail alone, and of launched levels."""
    import torch

    from beamtracer_b200 import _lib
    from beamtracer_b200.poisson import IonOpticsPoisson

    mesh = _plates(shape) if shape[0] < 50 else _three_plates(shape, 0.2e-3)
    solver = IonOpticsPoisson(mesh)
    solver.set_options(staged=staged)
    n = int(np.prod(shape))
    b = torch.from_numpy(np.random.default_rng(5).normal(size=n)).cuda()
    b[torch.from_numpy(mesh.fixed.reshape(-1)).cuda()] = 0.0
    _lib.context()

    def cycle(source, target):
        _lib.check(_lib.lib().bt_poisson_vcycle(solver._handle, _lib.dptr(source), None, 0,
                                                _lib.dptr(target)))  # fmt: skip

    expected = torch.empty_like(b)
    cycle(b, expected)
    for shift in (0, 1, shape[1], n - 1):
        for forward in (True, False):
            store = torch.zeros(2 * n, dtype=torch.float64, device="cuda")
            at, to = (0, shift) if forward else (shift, 0)
            store[at:at + n] = b
            cycle(store[at:at + n], store[to:to + n])
            assert torch.equal(store[to:to + n], expected), (shift, forward)
