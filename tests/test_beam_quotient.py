"""The beam frames' quotients (a reciprocal and one residual correction) round as
divisions do."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "finetoolsflexstructures.jl_gb300", "csrc")


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("quotient") / "libquotient.so")
    subprocess.run(["g++", "-O2", "-fPIC", "-shared", "-std=c++17", "-ffp-contract=off", "-I", CSRC, "-o", so,
                    os.path.join(HERE, "hostcheck", "quotientcheck.cpp")], check=True)
    L = ctypes.CDLL(so)
    L.qc_different.restype = ctypes.c_int64
    return L


@pytest.mark.parametrize("span", [0, 1, 60, 400])
def test_rounds_as_a_division(lib, span):
    rng = np.random.default_rng(span)
    n = 200_000
    a, b = (rng.uniform(1, 2, n) * rng.choice([-1, 1], n) * 2.0 ** rng.integers(-span, span + 1, n) for _ in range(2))
    # components of a vector over its length among them, and ones close to a power of two
    a[: n // 4] = b[: n // 4] * rng.uniform(-1, 1, n // 4)
    b[n // 4: n // 2] = 2.0 - rng.integers(0, 50, n // 4) * 2.0 ** -52
    P = lambda v: v.ctypes.data_as(ctypes.c_void_p)
    assert lib.qc_different(ctypes.c_int64(n), P(a), P(b)) == 0
