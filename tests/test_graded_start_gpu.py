"""Traces that start anywhere along a graded axis, against the oracle."""

from __future__ import annotations

import numpy as np
import pytest

from tests.golden.cases import TRACE_CHARGE, TRACE_OUTPUTS, copy_args
from tests.gpu_util import to_device, to_host

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("window", [1, 64])
@pytest.mark.parametrize("nx", [2, 3, 4, 33, 1025, 20_001])
def test_first_cell_on_a_graded_axis(nx, window):
    """The oracle's bits, for starts at nodes, the axis' ends and beyond, one representable
    number to either side of a node, and in cells of every part of the axis (where each window
    finds a trajectory's first cell)."""
    from beamtracer_b200.kernels import KERNELS
    from oracle import kernels as oracle

    rng = np.random.default_rng(nx)
    ny, h, n = 5, 1e-4, 97
    nodes = h * (np.arange(nx) + 0.4 * np.sin(0.7 * np.arange(nx)))
    nodes -= nodes[0]
    picked = nodes[rng.integers(0, nx, 24)]
    x, v = np.zeros((3, n)), np.zeros((3, n))
    x[0] = rng.uniform(-0.5 * h, nodes[-1] + 0.5 * h, n)
    x[0, :72] = np.concatenate([picked, np.nextafter(picked, -1.0), np.nextafter(picked, 1.0)])
    x[0, 72:77] = [0.0, nodes[-1], nodes[-2], -h, nodes[-1] + h]
    x[1] = rng.uniform(0.1, 0.9, n) * (ny - 1) * h
    v[0], v[1] = rng.choice([-3e5, 3e5], n), rng.uniform(-1e4, 1e4, n)
    capacity = 4
    args = [np.arange(n), x, v, np.full(n, 9.58e7), rng.uniform(0.5, 1.5, n), np.zeros(n, np.int64),
            np.full(n, -1), np.full(n, -1), rng.normal(size=(nx + 1) * ny) * 1e5,
            rng.normal(size=nx * (ny + 1)) * 1e5, np.array([[nx, ny, 0, 0, 0, 0]]),
            np.array([[0.0, 0.0, h, 0.0, 0.0, (nx - 1) * h, (ny - 1) * h]]), 0.0, 0.0, h,
            (nx - 1) * h, (ny - 1) * h, 0, 0, 0.5, 100, np.full((nx - 1, ny - 1), -1),
            np.zeros(1, np.int64), 1, np.array([0.5 * nodes[-1]]), np.zeros((n, 1, capacity, 8)),
            np.zeros((n, 1), np.int64), np.full(n, -1), np.zeros((1, 1, 2)), np.zeros(1, np.int64),
            1, np.zeros((1, nx * ny)), 1, nodes, 0.0]  # fmt: skip
    expected = copy_args(args)
    oracle.trace_trajectories_2d(*expected)
    device = to_device(args)
    KERNELS["trace_trajectories_2d"](*device, window=window)
    result = to_host(device)
    for key, i in TRACE_OUTPUTS.items():
        np.testing.assert_array_equal(result[i], expected[i], err_msg=key)
    total = expected[TRACE_CHARGE].sum(0)
    np.testing.assert_allclose(result[TRACE_CHARGE][0], total, rtol=0,
                               atol=1e-12 * np.abs(total).max())  # fmt: skip
