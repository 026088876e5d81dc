"""Traces whose steps the acceleration limits: starting at rest, and turning back."""

from __future__ import annotations

import numpy as np
import pytest

from tests.golden.cases import TRACE_CHARGE, TRACE_OUTPUTS, copy_args
from tests.gpu_util import load_golden, to_device, to_host

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("start", ["rest", "slow", "turning"])
@pytest.mark.parametrize("name", ["c0_i0_r0_g0_rel0", "c0_i1_r0_g0_rel0", "c1_i0_r0_g0_rel0",
                                  "c1_i1_r0_g0_rel0", "c2_i0_r0_g0_rel0", "c0_i0_r1_g1_rel0",
                                  "c1_i1_r1_g0_rel1"])  # fmt: skip
def test_steps_limited_by_the_acceleration(name, start):
    """The oracle's bits, for beams whose trajectories are at rest, nearly so, or turn back
    somewhere of their own (the charges, summed in another order, to 1e-12 of the largest)."""
    from beamtracer_b200.kernels import KERNELS
    from oracle import kernels as oracle

    args, _ = load_golden("trace_" + name)
    x, v, qm, upper_x = args[1], args[2], args[3], args[15]
    n = x.shape[1]
    rng = np.random.default_rng(n)
    field = 1e5 * (-1.0 if start == "turning" else 1.0)
    args[8][:] = field * (1.0 + 0.05 * rng.normal(size=args[8].size))
    args[9][:] = 0.02 * field * rng.normal(size=args[9].size)
    x[0] = rng.uniform(0.0, 0.3 * upper_x, n)
    v[:] = 0.0
    if start == "slow":
        v[:] = rng.normal(size=v.shape) * 10.0 ** rng.uniform(-6.0, 3.0, n)
    if start == "turning":
        v[0] = np.sqrt(2.0 * np.abs(qm * field) * upper_x) * rng.uniform(0.05, 0.8, n)
        v[1] = 0.05 * v[0] * rng.normal(size=n)
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


@pytest.mark.parametrize("start", ["rest", "slow", "turning"])
@pytest.mark.parametrize("name", ["i0_r0_m0_b0_j0", "i0_r0_m1_b1_j1", "i1_r0_m0_b0_j0",
                                  "i1_r0_m1_b1_j1"])  # fmt: skip
def test_3d_steps_limited_by_the_acceleration(name, start):
    """The same in three dimensions (charge and current within 1e-13 of the largest)."""
    from beamtracer_b200.kernels import KERNELS
    from oracle.trace3d import trace_trajectories_3d

    args, _ = load_golden("trace3d_" + name)
    x, v, qm, upper_x = args[1], args[2], args[3], args[19]
    n = x.shape[1]
    rng = np.random.default_rng(n)
    field = 1e5 * (-1.0 if start == "turning" else 1.0)
    args[8][:] = field * (1.0 + 0.05 * rng.normal(size=args[8].size))
    for i in (9, 10):
        args[i][:] = 0.02 * field * rng.normal(size=args[i].size)
    x[0] = rng.uniform(0.0, 0.3 * upper_x, n)
    v[:] = 0.0
    if start == "slow":
        v[:] = rng.normal(size=v.shape) * 10.0 ** rng.uniform(-6.0, 3.0, n)
    if start == "turning":
        v[0] = np.sqrt(2.0 * np.abs(qm * field) * upper_x) * rng.uniform(0.05, 0.8, n)
        v[1:] = 0.05 * v[0] * rng.normal(size=(2, n))
    expected = copy_args(args)
    trace_trajectories_3d(*expected)
    device = to_device(args)
    KERNELS["trace_trajectories_3d"](*device)
    result = to_host(device)
    for i in (1, 2, 5, 6, 7, 31, 32, 34, 35):
        np.testing.assert_array_equal(result[i], expected[i], err_msg=f"argument {i}")
    for i in (37, 39) if args[38] else (37,):
        want = expected[i].sum(axis=0)
        assert float(np.abs(result[i].sum(axis=0) - want).max()) <= 1e-13 * float(np.abs(want).max())
