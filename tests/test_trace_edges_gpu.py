"""Traces whose points leave the mesh on every side, near and far, against the oracle."""

from __future__ import annotations

import numpy as np
import pytest

from tests.golden.cases import TRACE_CHARGE, TRACE_OUTPUTS, copy_args
from tests.gpu_util import load_golden, to_device, to_host

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fraction", [0.5, 1.7, 40.0])
@pytest.mark.parametrize("name", ["c0_i0_r0_g0_rel0", "c0_i1_r0_g0_rel0", "c0_i0_r1_g0_rel1",
                                  "c1_i0_r0_g0_rel0", "c1_i1_r1_g1_rel1", "c2_i0_r0_g0_rel0",
                                  "c2_i0_r1_g1_rel0"])  # fmt: skip
def test_points_past_every_edge(name, fraction):
    """Trajectories towards, along and past the four edges, from within the mesh and from
    outside it, at steps of part of a cell to many cells: the oracle's bits (the charges,
    summed in another order, to 1e-12 of the largest)."""
    from beamtracer_b200.kernels import KERNELS
    from oracle import kernels as oracle

    args, _ = load_golden("trace_" + name)
    x, v = args[1], args[2]
    h, upper_x, upper_y = args[14], args[15], args[16]
    n = x.shape[1]
    rng = np.random.default_rng(n + len(name))
    far = 1e10 * h  # (cells past 2^31)
    x[0] = rng.uniform(0.0, upper_x, n)
    x[1] = rng.uniform(0.0, upper_y, n)
    x[2] *= 0.01
    picks = [-far, -3.3 * h, -h, -0.5 * h, -1e-9 * h, 0.0, 0.5 * h, upper_x - 0.5 * h, upper_x,
             upper_x + 0.5 * h, upper_x + h, upper_x + far]  # fmt: skip
    x[0, :24] = rng.permutation(np.tile(picks, 2))
    x[1, 12:36] = rng.permutation(np.tile([p if p < upper_x - h else p - upper_x + upper_y
                                           for p in picks], 2))  # fmt: skip
    angle = rng.uniform(0.0, 2.0 * np.pi, n)
    angle[::3] = np.round(angle[::3] / (0.5 * np.pi)) * 0.5 * np.pi  # along an axis
    speed = np.hypot(v[0], v[1])
    v[0], v[1] = speed * np.cos(angle), speed * np.sin(angle)
    args[19] = fraction
    expected = copy_args(args)
    oracle.trace_trajectories_2d(*expected)
    device = to_device(args)
    device[TRACE_CHARGE] = device[TRACE_CHARGE][:1].clone()
    KERNELS["trace_trajectories_2d"](*device)
    result = to_host(device)
    for key, i in TRACE_OUTPUTS.items():
        np.testing.assert_array_equal(result[i], expected[i], err_msg=key)
    total = expected[TRACE_CHARGE].sum(0)
    np.testing.assert_allclose(result[TRACE_CHARGE][0], total, rtol=0,
                               atol=1e-12 * np.abs(total).max())  # fmt: skip
