"""The tracer's square roots and quotients without a branch (``Num`` in ``csrc/common.cuh``).

The same steps in C, with the C library's ``fma`` and with reciprocals and reciprocal roots
perturbed by up to 2^-18.9 in place of the hardware's approximations (at most 2^-19 off),
must give ``sqrt(s)``, ``a / b`` and ``p / sqrt(s)`` bit for bit: on random significands, on
the coordinates and speeds a trace meets, and on every significand whose root lies so near
to a rounding boundary that the last correction could fall on its other side (s = M^2 + M + c
scaled, |c| < 256).  The device code itself is checked by the bit-exact trace parity tests.
"""

from __future__ import annotations

import ctypes
import shutil
import subprocess

import numpy as np
import pytest

SOURCE = r"""
#include <math.h>
#include <stdint.h>
#include <string.h>

static double root(double s, double d, double *y) {
    const double y0 = (1.0 / sqrt(s)) * (1.0 + d);
    const double e = fma(-(s * y0), y0, 1.0);
    *y = fma(fma(0.375, e, 0.5), e * y0, y0);
    const double g = s * *y;
    return fma(fma(-g, g, s), 0.5 * *y, g);
}
static double inverse_from(double b, double y) {
    y = fma(fma(-b, y, 1.0), y, y);
    return fma(fma(-b, y, 1.0), y, y);
}
static double inverse(double b, double d) {
    const double y = (1.0 / b) * (1.0 + d);
    const double e = fma(-b, y, 1.0);
    return inverse_from(b, fma(fma(e, e, e), y, y));
}
static double over(double a, double b, double rb) {
    double q = a * rb;
    q = fma(fma(-q, b, a), rb, q);
    return fma(fma(-q, b, a), rb, q);
}
/* the bit patterns that differ: roots, quotients by roots, quotients */
void mismatches(const double *s, const double *a, const double *d, long n, long *bad) {
    for (long i = 0; i < n; ++i) {
        double y;
        const double r = root(s[i], d[i], &y), e = sqrt(s[i]);
        if (memcmp(&r, &e, sizeof r)) ++bad[0];
        uint64_t bits;
        memcpy(&bits, &e, sizeof bits);
        if ((uint32_t)bits != 0xffffffffu) {
            const double q = over(a[i], e, inverse_from(e, y)), w = a[i] / e;
            if (memcmp(&q, &w, sizeof q)) ++bad[1];
        }
        memcpy(&bits, &s[i], sizeof bits);
        if ((uint32_t)bits != 0xffffffffu) {
            const double q = over(a[i], s[i], inverse(s[i], d[i])), w = a[i] / s[i];
            if (memcmp(&q, &w, sizeof q)) ++bad[2];
        }
    }
}
"""


@pytest.fixture(scope="module")
def mismatches(tmp_path_factory):
    gcc = shutil.which("gcc")
    if gcc is None:
        pytest.skip("no C compiler")
    d = tmp_path_factory.mktemp("roots")
    (d / "roots.c").write_text(SOURCE)
    subprocess.run([gcc, "-O2", "-ffp-contract=off", "-shared", "-fPIC", "-o", str(d / "roots.so"),
                    str(d / "roots.c"), "-lm"], check=True)  # fmt: skip
    lib = ctypes.CDLL(str(d / "roots.so"))

    def count(s, a, seed_error):
        out = (ctypes.c_long * 3)()
        arrays = [np.ascontiguousarray(v, dtype=float) for v in (s, a, seed_error)]
        lib.mismatches(*(v.ctypes.data_as(ctypes.c_void_p) for v in arrays),
                       ctypes.c_long(arrays[0].size), out)  # fmt: skip
        return list(out)

    return count


def near_boundary() -> np.ndarray:
    """Every double in [1, 4) that is M^2 + M + c, scaled, for a 53-bit M and even |c| < 256."""
    found = []
    for bits in (52, 53):  # the double's last place in units of the square's
        for c in range(-256, 257, 2):
            for root in (0, 1):
                for b in range(1, bits):  # lift the root of M^2 + M + c = 0 mod 2^(b + 1)
                    if (root * root + root + c) % (1 << (b + 1)):
                        root |= 1 << b
                for m in range(root, 1 << 53, 1 << bits):
                    t = (m * m + m + c) >> bits
                    if m >= 1 << 52 and (t < 1 << 53 or (t < 1 << 54 and t % 2 == 0)):
                        found.append(float(t) * 2.0 ** (bits - 104))
    return np.array(found)


def test_random_operands(mismatches):
    rng = np.random.default_rng(0)
    n = 400_000
    s = np.ldexp(rng.uniform(1.0, 2.0, n), rng.integers(-300, 300, n))
    a = np.ldexp(rng.uniform(-2.0, 2.0, n), rng.integers(-90, 90, n))
    a[::17] = 0.0
    assert mismatches(s, a, rng.uniform(-2.0**-18.9, 2.0**-18.9, n)) == [0, 0, 0]


def test_the_trace_s_operands(mismatches):
    """Squared radii and speeds, and the coordinates and spacings they divide."""
    rng = np.random.default_rng(1)
    n = 400_000
    s = np.where(rng.random(n) < 0.5, rng.uniform(0.0, 4e-4, n), rng.uniform(1e8, 1e14, n))
    a = np.where(rng.random(n) < 0.5, rng.uniform(-2e-2, 2e-2, n), 1e-4)
    assert mismatches(s, a, rng.uniform(-2.0**-18.9, 2.0**-18.9, n)) == [0, 0, 0]


@pytest.mark.parametrize("error", [-(2.0**-18.9), -(2.0**-22), 0.0, 2.0**-20, 2.0**-18.9])
def test_roots_nearest_to_a_rounding_boundary(mismatches, error):
    base = near_boundary()
    assert base.size > 500
    s = np.concatenate([np.ldexp(base, e) for e in (-300, -20, 0, 2, 40, 300)])
    assert mismatches(s, np.ones(s.size), np.full(s.size, error))[0] == 0
