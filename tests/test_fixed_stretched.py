"""Accuracy of the FS_FP64 elements on stretched triangles: the fixed point
(csrc/fs_elem_fixed.cuh) and the double arithmetic that it stands for, both
against the same element in long double, over shapes from equilateral to the
longest that the fixed point takes, axis-aligned plates and tilted ones.

Elongation is the longest edge squared over twice the area.  The energies are
u' dK u of nine linear and quadratic displacement modes u.  Bound: in the mean
(of the logarithm) over each factor of two of elongation, the fixed point's
error of every energy and of K_ij against sqrt(K_ii K_jj) is at most sqrt(2)
times the double arithmetic's, half a bit."""
import ctypes
import os
import re
import subprocess

import numpy as np
import pytest

from flexshell import _abi, materials
from flexshell._lib import ptr

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "finetoolsflexstructures.jl_gb300", "csrc")
LONGEST = 32.0


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    if np.finfo(np.longdouble).nmant < 60:
        pytest.skip("long double is no wider than double")
    d = tmp_path_factory.mktemp("stretch")
    src = open(os.path.join(CSRC, "fs_elem_math.cuh")).read()
    src = re.sub(r"\bdouble\b", "long double", src)
    src = src.replace("namespace fs ", "namespace fsl ").replace("sizeof(R) == 8", "sizeof(R) >= 8")
    for f in ("sqrt", "sin", "cos"):
        src = re.sub(r"(?<![\w.])%s\(" % f, f + "l(", src)
    (d / "wide_elem_math.h").write_text(src)
    so = str(d / "libstretch.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-w", "-fno-strict-aliasing", "-I", CSRC, "-I", str(d),
                    "-I", os.path.join(os.path.dirname(HERE), "include"), "-o", so,
                    os.path.join(HERE, "hostcheck", "stretchcheck.cpp")], check=True)
    return ctypes.CDLL(so)


def _elongation(P):
    e = [P[:, (i + 1) % 3] - P[:, i] for i in range(3)]
    return np.max([(v ** 2).sum(1) for v in e], axis=0) / np.abs(e[0][:, 0] * e[1][:, 1] - e[0][:, 1] * e[1][:, 0])


def triangles(n, lo, hi, flat, seed):
    """n triangles of elongation lo to hi: nodes in the plane, frames, coordinates,
    normals and thicknesses."""
    rng = np.random.default_rng(seed)
    P = np.zeros((0, 3, 2))
    while len(P) < n:
        Q = rng.uniform(-1, 1, (200 * n, 3, 2))
        Q[:, :, 1] *= 2.0 ** -rng.uniform(0, np.log2(hi), 200 * n)[:, None]
        e = _elongation(Q)
        P = np.concatenate([P, Q[(e >= lo) & (e < hi)]])
    P = P[:n] * 10.0 ** rng.uniform(-2, 0, n)[:, None, None]
    R = np.broadcast_to(np.eye(3), (n, 3, 3))
    if not flat:
        R, _ = np.linalg.qr(rng.normal(size=(n, 3, 3)))
        R = R * np.sign(np.linalg.det(R))[:, None, None]
    X = np.einsum("eai,eic->eac", P, R[:, :2])
    N = np.repeat(R[:, None, 2], 3, axis=1) + (0.0 if flat else 0.03) * rng.uniform(-1, 1, (n, 3, 3))
    N /= np.linalg.norm(N, axis=2, keepdims=True)
    t = np.abs(P).max(axis=(1, 2)) * 10.0 ** rng.uniform(-3, -1, n)
    return X, R, N, t


def modes(X, R):
    """Nine displacement fields at the nodes, in the element plane's axes."""
    n = len(X)
    x, y, _ = np.moveaxis(np.einsum("eac,eic->eai", X - X.mean(axis=1, keepdims=True), R), 2, 0)
    o, one = np.zeros_like(x), np.ones_like(x)
    local = [(x, o, o, o, o, o), (o, y, o, o, o, o), (y / 2, x / 2, o, o, o, o),
             (o, o, -x * x / 2, o, x, o), (o, o, -y * y / 2, -y, o, o), (o, o, -x * y, -x, y, o),
             (o, o, o, o, one, o), (o, o, o, one, o, o), (o, o, o, o, x, o)]
    u = np.array(local).transpose(0, 2, 3, 1)   # mode, element, node, component
    g = np.concatenate([np.einsum("meai,eic->meac", u[..., :3], R), np.einsum("meai,eic->meac", u[..., 3:], R)], axis=3)
    return g.reshape(9, n, 18)


def run(lib, X, N, t, layered=False):
    n = len(X)
    Dps, Dt = materials.shell_material_stiffness(materials.MatDeforElastIso(2.0e11, 0.3, 7850.0))
    p = _abi.make_params(Dps, Dt, 7850.0, 0.0, quads=False, drilling_stiffness_scale=1.0)
    K, F, D = (np.zeros((n, 18, 18)) for _ in range(3))
    far = np.zeros(n, np.uint8)
    a = [np.ascontiguousarray(v) for v in (X, N, t)]
    assert lib.stretched_triangles(ctypes.c_int64(n), *[ptr(v) for v in a], ctypes.byref(p), ptr(K), ptr(F), ptr(D), ptr(far)) == 0
    return K, F, D, far.astype(bool)


def ratios(K, F, D, X, R):
    """Mean ratios of the errors: of K_ij (worst of each element), of nine energies."""
    s = np.sqrt(np.maximum(np.einsum("eii->ei", K), 0.0))
    s = s[:, :, None] * s[:, None, :]
    s[s == 0] = np.inf
    tiny = 1e-18
    out = [np.log((np.abs(F / s).max(axis=(1, 2)) + tiny) / (np.abs(D / s).max(axis=(1, 2)) + tiny)).mean()]
    for u in modes(X, R):
        en = np.einsum("ei,eij,ej->e", u, K, u)
        f, d = (np.abs(np.einsum("ei,eij,ej->e", u, E, u) / en) + tiny for E in (F, D))
        out.append(np.log(f / d).mean())
    return np.exp(out)


@pytest.mark.parametrize("flat", [True, False])
@pytest.mark.parametrize("lo", [1.0, 2.0, 4.0, 8.0, 16.0])
def test_no_further_off_than_double(lib, lo, flat):
    X, R, N, t = triangles(500, lo, 2 * lo, flat, int(lo))
    K, F, D, far = run(lib, X, N, t)
    assert not far.any()
    r = ratios(K, F, D, X, R)
    assert (r <= 2 ** 0.5).all(), r


@pytest.mark.parametrize("flat", [True, False])
def test_longer_triangles_are_left_to_the_double_kernel(lib, flat):
    X, R, N, t = triangles(300, LONGEST * (1 + 1e-9), 1e4, flat, 3)
    assert run(lib, X, N, t)[3].all()
