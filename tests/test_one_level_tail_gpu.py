"""A multigrid tail of the coarsest level alone: the cluster's first block sends its
right-hand side to the other blocks almost as soon as it starts."""

from __future__ import annotations

import numpy as np
import pytest

from oracle import poisson as oracle
from tests.test_poisson_gpu import _plates, _three_plates

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(41, 21), (257, 65), (64, 33)], ids=str)
def test_one_level_tail(shape):
    """The V-cycle whose tail is the coarsest level (of at most 256 nodes) equals the one whose
    coarsest level has a launch of its own, to the rounding of a sum of 256 products (1e-12 of
    the largest value), on every one of many launches behind one another; and the solve meets
    the oracle's LU to 1e-9 of the plates' voltage."""
    import torch

    from beamtracer_b200 import _lib
    from beamtracer_b200.poisson import IonOpticsPoisson

    mesh = _plates(shape) if shape[0] < 50 else _three_plates(shape, 0.2e-3)
    nodes = int(np.prod(shape))
    while nodes > 256:
        shape = tuple(n // 2 + 1 if n > 3 else n for n in shape)
        nodes = int(np.prod(shape))
    rng = np.random.default_rng(2)
    b = torch.from_numpy(rng.uniform(size=mesh.shape)).cuda()
    b[torch.from_numpy(mesh.fixed).cuda()] = 0.0
    rho = rng.uniform(0.0, 1e-5, mesh.shape)
    expected = oracle.solve(oracle.operator_of_mesh(mesh), rho)
    cycles = []
    for tail_nodes in (1, nodes):
        solver = IonOpticsPoisson(mesh)
        solver.set_options(tail_nodes=tail_nodes)
        np.testing.assert_allclose(solver.solve(rho), expected, rtol=0,
                                   atol=1e-9 * max(np.ptp(expected), 1.0))  # fmt: skip
        _lib.context()
        out = [torch.empty_like(b) for _ in range(50)]
        for z in out:
            _lib.check(_lib.lib().bt_poisson_vcycle(solver._handle, _lib.dptr(b), None, 0,
                                                    _lib.dptr(z)))  # fmt: skip
        assert all(torch.equal(z, out[0]) for z in out)
        cycles.append(out[0])
    own, tail = cycles
    assert float((tail - own).abs().max()) <= 1e-12 * float(own.abs().max())
