"""The FS_FP64 elements' fixed point on the host: its numbers against exact
arithmetic and its element matrices against the same elements in double
(csrc/fs_elem_fixed.cuh and csrc/fs_elem_math.cuh built by a host compiler),
over shapes, sizes, orientations, thicknesses and normals, and the elements it
leaves to the double path.

Tolerances.  A number kept in a group of exponent E is off by at most 2^(E-57)
(58 bits, cut), a dot product of m terms of two groups by m (2 + 1) 2^(E+E'-58)
more than its last rounding (two cut factors and the dropped low products).
Element matrices: 1e-12 of the largest entry, the repository's FP64 parity
bound."""
import ctypes
import os
import subprocess
from fractions import Fraction

import numpy as np
import pytest

from flexshell import _abi, materials
from flexshell._lib import ptr

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("fixed") / "libfixedcheck.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-w", "-ffp-contract=off",
                    "-I", os.path.join(ROOT, "finetoolsflexstructures.jl_gb300", "csrc"),
                    "-I", os.path.join(ROOT, "include"), "-o", so, os.path.join(HERE, "hostcheck", "fixedcheck.cpp")],
                   check=True)
    return ctypes.CDLL(so)


def _elements(nen, n, seed, shape=0.25, warp=0.0, tilt=0.1, thin=(-3.5, -0.5), size=(-4, 2), flat=False):
    """n random elements: base triangle or square with its nodes moved by
    `shape`, out of plane by `warp`, normals tilted, t / h and h log-uniform."""
    rng = np.random.default_rng(seed)
    base = np.array([[0, 0], [1, 0], [0, 1.0]] if nen == 3 else [[0, 0], [1, 0], [1, 1], [0, 1.0]])
    P = np.zeros((n, nen, 3))
    P[:, :, :2] = base + shape * rng.uniform(-1, 1, (n, nen, 2))
    P[:, :, 2] = warp * rng.uniform(-1, 1, (n, nen))
    Q, _ = np.linalg.qr(rng.normal(size=(n, 3, 3)))
    Q *= np.sign(np.linalg.det(Q))[:, None, None]
    if flat:
        Q[:] = np.eye(3)
    h = 10.0 ** rng.uniform(*size, n)
    X = np.einsum("eij,eaj->eai", Q, P + np.r_[rng.uniform(-5, 5, 2), 0.0]) * h[:, None, None]
    N = np.zeros((n, nen, 3))
    N[:, :, 2] = 1.0
    N += tilt * rng.uniform(-1, 1, (n, nen, 3)) * (not flat)
    N = np.einsum("eij,eaj->eai", Q, N)
    N /= np.linalg.norm(N, axis=2, keepdims=True)
    valid = (rng.uniform(size=(n, nen)) < 0.9).astype(np.uint8)
    t = h * 10.0 ** rng.uniform(*thin, n)
    return X, N, valid, t


def _run(lib, nen, X, N, valid, t, scale=1.0):
    n, nd = len(X), 6 * nen
    Dps, Dt = materials.shell_material_stiffness(materials.MatDeforElastIso(2.0e11, 0.3, 7850.0))
    p = _abi.make_params(Dps, Dt, 7850.0, 0.0, quads=nen == 4, drilling_stiffness_scale=scale)
    K, D, ok = np.zeros((n, nd, nd)), np.zeros((n, nd, nd)), np.zeros(n, np.uint8)
    a = [np.ascontiguousarray(v) for v in (X, N, valid, t)]
    assert lib.fixed_elements(nen, ctypes.c_int64(n), *[ptr(v) for v in a], ctypes.byref(p), ptr(K), ptr(D), ptr(ok)) == 0
    return K, D, ok.astype(bool)


@pytest.mark.parametrize("nen", [3, 4])
@pytest.mark.parametrize("kind", ["plain", "flat", "thin", "thick", "folded", "stretched", "scale0", "scale1e3"])
def test_element_matrices_match_the_double_path(lib, nen, kind):
    kw = {"plain": {}, "flat": dict(flat=True), "thin": dict(thin=(-6, -4)), "thick": dict(thin=(-0.5, 0.5)),
          "folded": dict(tilt=1.0, warp=0.1 * (nen == 4)), "stretched": dict(shape=0.45)}.get(kind, {})
    X, N, valid, t = _elements(nen, 400, 7, **kw)
    scale = {"scale0": 0.0, "scale1e3": 1e3}.get(kind, 1.0)
    K, D, ok = _run(lib, nen, X, N, valid, t, scale)
    assert ok.all()
    assert np.isfinite(K).all()
    mx = np.abs(D).max(axis=(1, 2))
    assert (np.abs(K - D).max(axis=(1, 2)) <= 1e-12 * mx).all()
    assert np.array_equal(K, K.transpose(0, 2, 1))
    if kind == "flat":
        # membrane and bending uncoupled: the same exact zeros
        assert np.array_equal(K == 0, D == 0)


@pytest.mark.parametrize("nen", [3, 4])
def test_elements_left_to_the_double_path(lib, nen):
    X, N, valid, t = _elements(nen, 9, 3)
    valid[:] = 1
    X[0, 1] = X[0, 0]                                        # a zero first edge (T3), a collapsed side (Q4)
    X[1] = X[1, :1] + np.arange(nen)[:, None] * np.ones(3)   # all nodes on a line
    X[2, 0, 0] = np.nan
    X[3, 0, 0] = np.inf
    N[4, 1] = np.nan
    t[5] = np.nan
    X[6] *= 1e-90
    X[7] *= 1e90
    K, D, ok = _run(lib, nen, X, N, valid, t)
    assert ok[8] and np.isfinite(K[8]).all()
    assert not ok[1:8].any()
    assert not ok[0] or nen == 4


def test_numbers_and_dot_products(lib):
    rng = np.random.default_rng(1)
    for E in (-150, -3, 0, 1, 40, 190):
        x = np.ldexp(rng.uniform(-1, 1, 500), E - rng.integers(0, 70, 500).astype(int))
        x[:4] = [0.0, -0.0, np.ldexp(1.0, E - 1), -np.ldexp(1.0, E - 58)]
        out = np.zeros_like(x)
        lib.fixed_round_trip(ctypes.c_int64(x.size), ptr(x), E, ptr(out))
        assert (np.abs(out - x) <= np.ldexp(1.0, E - 57) + np.abs(x) * 2.0 ** -53).all()
    for m in (1, 2, 3, 9, 12):
        ea, eb = 3, -7
        a = np.ldexp(rng.uniform(-1, 1, (300, m)), ea)
        b = np.ldexp(rng.uniform(-1, 1, (300, m)), eb)
        a[:, -1] *= 1e-6
        if m > 1:
            b[:50, 0] = -(a[:50, 1:] * b[:50, 1:]).sum(1) / a[:50, 0]      # cancelling sums
            b[:50, 0] = np.clip(b[:50, 0], -np.ldexp(0.99, eb), np.ldexp(0.99, eb))
        out = np.zeros(300)
        lib.fixed_dots(ctypes.c_int64(300), m, ptr(np.ascontiguousarray(a)), ptr(np.ascontiguousarray(b)), ea, eb, ptr(out))
        for i in range(300):
            want = sum((Fraction(p) * Fraction(q) for p, q in zip(a[i].tolist(), b[i].tolist())), Fraction(0))
            bound = Fraction(3 * m, 1) * Fraction(2) ** (ea + eb - 58) + Fraction(2) ** (ea + eb - 57) + abs(want) / 2 ** 53
            assert abs(Fraction(float(out[i])) - want) <= bound
