"""The 64-bit sums of the fixed point (csrc/fs_fixed.cuh on the host) at the
largest entries and the longest sums that the element kernels form, all of one
sign and of mixed signs, against exact arithmetic.

Bound: each factor is cut by less than 2^-58 of its group's exponent, a product
drops at most 2^-60 of it, the sum is cut once and rounded once: m terms of
factors up to c and c' are off by at most m (c + c' + 1) + 2 units of 2^(E-58),
beside half the last bit of the result."""
import ctypes
from fractions import Fraction

import numpy as np
import pytest

from flexshell._lib import ptr
from test_fixed_elements import lib  # noqa: F401

# name: largest entries, products
SUMS = {"M triangle": (1.9999, 1.9999, 3), "M quad": (0.9999, 0.9999, 12), "T triangle": (1.2, 1.2, 5),
        "T quad": (1.2, 1.2, 20), "R triangle": (1.4143, 1.4143, 5), "R quad": (0.7072, 0.7072, 20),
        "TR triangle": (1.2, 1.4143, 5), "TR quad": (1.2, 0.7072, 20), "layered triangle": (0.9999, 0.9999, 13),
        "layered quad": (0.5, 0.5, 33), "drilling": (0.9999, 0.9999, 1)}


@pytest.mark.parametrize("name", sorted(SUMS))
def test_longest_sums_of_the_largest_entries(lib, name):  # noqa: F811
    ca, cb, m = SUMS[name]
    assert ca * cb * m < 32
    ea, eb = 3, -7
    rng = np.random.default_rng(m)
    n = 200
    a = np.ldexp(ca * (1 - 1e-3 * rng.uniform(0, 1, (n, m)) ** 4), ea)
    b = np.ldexp(cb * (1 - 1e-3 * rng.uniform(0, 1, (n, m)) ** 4), eb)
    a[n // 2:] *= rng.choice([-1, 1], (n - n // 2, m))     # mixed signs
    a[: n // 4] = np.ldexp(ca, ea)                          # the very largest
    b[: n // 8] = np.ldexp(cb, eb)
    a[n // 8: n // 4] *= -1
    out = np.zeros(n)
    lib.fixed_dots(ctypes.c_int64(n), m, ptr(np.ascontiguousarray(a)), ptr(np.ascontiguousarray(b)), ea, eb, ptr(out))
    unit = Fraction(2) ** (ea + eb - 58)
    for i in range(n):
        want = sum((Fraction(p) * Fraction(q) for p, q in zip(a[i].tolist(), b[i].tolist())), Fraction(0))
        bound = (m * Fraction(ca + cb + 1) + 2) * unit + abs(want) / 2 ** 53
        assert abs(Fraction(float(out[i])) - want) <= bound
