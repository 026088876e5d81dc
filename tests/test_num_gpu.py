"""The device's straight-line roots and quotients (``Num<true>`` in ``csrc/common.cuh``).

A kernel compiled here from that header applies them to arrays.  Where ``odd()`` is false they
must be ``sqrt(s)``, ``a / sqrt(s)`` and ``a / s`` bit for bit (numpy's, which round to nearest;
a zero dividend gives +0); ``odd()`` must be true for every operand, a zero root or dividend
apart, outside 2^-401 .. 2^401, and false inside 2^-399 .. 2^399 unless the divisor's low word is
all ones.
"""

from __future__ import annotations

import ctypes
import subprocess

import numpy as np
import pytest

from tests.test_exact_roots import near_boundary

pytestmark = pytest.mark.gpu

SOURCE = r"""
#include "common.cuh"

__global__ void apply(const double *s, const double *a, long n, double *out, uint8_t *odd) {
    const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    bt::Num<true> of_root, by_root, by_value;
    out[i] = of_root.root(s[i]);
    double y;
    const double r = by_root.root(s[i], y);
    out[n + i] = by_root.over(a[i], r, by_root.inverse(r, y));
    out[2 * n + i] = by_value.div(a[i], s[i]);
    odd[i] = of_root.odd();
    odd[n + i] = by_root.odd();
    odd[2 * n + i] = by_value.odd();
}

extern "C" int run(const double *s, const double *a, long n, double *out, uint8_t *odd) {
    apply<<<(unsigned)((n + 255) / 256), 256>>>(s, a, n, out, odd);
    return (int)cudaDeviceSynchronize();
}
"""


@pytest.fixture(scope="module")
def num(tmp_path_factory):
    import torch

    from beamtracer_b200 import build

    d = tmp_path_factory.mktemp("num")
    (d / "num.cu").write_text(SOURCE)
    subprocess.run([build.nvcc(), *build.ARCH, *build.COMMON, "--fmad=false", f"-I{build.INCLUDE}",
                    f"-I{build.CSRC}", "-shared", "-o", str(d / "num.so"), str(d / "num.cu")],
                   check=True)  # fmt: skip
    run = ctypes.CDLL(str(d / "num.so")).run

    def apply(s, a):
        given = [torch.from_numpy(np.ascontiguousarray(v)).cuda() for v in (s, a)]
        out = torch.empty((3, s.size), dtype=torch.float64, device="cuda")
        odd = torch.empty((3, s.size), dtype=torch.uint8, device="cuda")
        torch.cuda.synchronize()
        pointers = [ctypes.c_void_p(t.data_ptr()) for t in (*given, out, odd)]
        assert run(*pointers[:2], ctypes.c_long(s.size), *pointers[2:]) == 0
        return out.cpu().numpy(), odd.cpu().numpy().astype(bool)

    return apply


def edges() -> np.ndarray:
    """Zero, subnormals, the ranges' ends, all-ones significands, infinity and no number."""
    ones = 2.0 - 2.0**-52
    low_ones = 1.0 + (2.0**32 - 1) * 2.0**-52
    values = [0.0, 5e-324, 2.0**-1050, 2.0**-1043, 2.0**-1042, 2.0**-1030, 2.0**-1022, 2.0**-1021,
              2.0**-600, 2.0**600, 2.0**1023, np.inf, np.nan]  # fmt: skip
    for e in (-402, -401, -400, -399, -1, 0, 1, 398, 399, 400, 401):
        values += [2.0**e, np.nextafter(2.0**e, 0.0), np.nextafter(2.0**e, np.inf),
                   ones * 2.0**e, low_ones * 2.0**e, 1.5 * 2.0**e]  # fmt: skip
    return np.array(values)


def check(num, s, a):
    out, odd = num(s, a)
    with np.errstate(all="ignore"):
        root = np.sqrt(s)
        expected = np.stack([root, a / root, a / s])

    def inside(v, margin, zero):
        m = np.abs(v)
        return ((m >= 2.0 ** -(400 - margin)) & (m <= 2.0 ** (400 - margin))) | (zero & (v == 0.0))

    def low_ones(v):
        return v.view(np.uint64) & 0xFFFFFFFF == 0xFFFFFFFF

    yes, no = np.ones(s.size, bool), np.zeros(s.size, bool)
    # by a zero root nothing is divided: its quotient is masked where it is asked for
    must_be = np.stack([~inside(s, -1, yes), ~inside(s, -1, yes), ~inside(s, -1, no)])
    small = (a != 0.0) & (np.abs(a) < 2.0**-401)
    must_be[1:] |= small
    may_not = np.stack([inside(s, 1, yes), inside(s, 1, no) & inside(a, 1, yes) & ~low_ones(root),
                        inside(s, 1, no) & inside(a, 1, yes) & ~low_ones(s)])  # fmt: skip
    assert np.all(odd[must_be])
    assert not np.any(odd[may_not])
    compared = ~odd
    compared[1] &= root != 0.0
    assert compared.sum() > 0
    assert np.array_equal(out[compared], expected[compared])


def test_edges(num):
    values = edges()
    s, a = (g.reshape(-1) for g in np.meshgrid(values, np.concatenate([values, -values])))
    keep = np.isfinite(a) & (np.abs(a) <= 2.0**401)  # (a huge dividend is its caller's to test)
    check(num, s[keep], a[keep])


def test_random_operands(num):
    rng = np.random.default_rng(0)
    n = 1_000_000
    s = np.ldexp(rng.uniform(1.0, 2.0, n), rng.integers(-399, 399, n))
    a = np.ldexp(rng.uniform(-2.0, 2.0, n), rng.integers(-399, 398, n))
    a[::17] = 0.0
    s[::19] = np.ldexp(rng.uniform(1.0, 2.0, s[::19].size), rng.integers(-1074, 1023, s[::19].size))
    check(num, s, a)


def test_roots_nearest_to_a_rounding_boundary(num):
    base = near_boundary()
    s = np.concatenate([np.ldexp(base, e) for e in (-300, -20, 0, 2, 40, 300)])
    check(num, s, np.ones(s.size))


TINY = [0.0, 5e-324, 2.0**-1050, 1e-310, 2.0**-1022, 1e-200, 1e-157, -1e-157, 2.0**-400, 1e-60]


@pytest.mark.parametrize("origin", [0.0, 2.0**-230, -(2.0**-100)])
@pytest.mark.parametrize("name", ["c0_i0_r0_g0_rel0", "c0_i1_r0_g0_rel0", "c1_i0_r0_g0_rel0",
                                  "c1_i1_r0_g0_rel0", "c2_i0_r0_g0_rel0", "c1_i0_r0_g1_rel0",
                                  "c1_i1_r1_g0_rel1"])  # fmt: skip
def test_traces_from_tiny_coordinates(name, origin):
    """Trajectories that start within a tiny distance of an axis, at rest across it or not, on
    meshes whose origin is zero or tiny: the oracle's bits (the charges, summed in another
    order, to 1e-12 of the largest)."""
    from beamtracer_b200.kernels import KERNELS
    from oracle import kernels as oracle
    from tests.golden.cases import TRACE_CHARGE, TRACE_OUTPUTS, copy_args
    from tests.gpu_util import load_golden, to_device, to_host

    args, _ = load_golden("trace_" + name)
    x, v = args[1], args[2]
    rng = np.random.default_rng(len(name))
    for axis in range(3):
        chosen = rng.random(x.shape[1]) < (0.8 if axis else 0.3)
        x[axis, chosen] = rng.choice(TINY, chosen.sum())
        if axis:
            v[axis, rng.random(x.shape[1]) < 0.7] = 0.0
    if origin and not args[32]:  # (a graded axis has its own first node)
        args[12] = args[13] = origin
        args[11][-1, 0] = args[11][-1, 1] = origin
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
