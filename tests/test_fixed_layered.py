"""Accuracy of the layered FS_FP64 elements, whose Gram products are in fixed
point (csrc/fs_elem_fixed.cuh): their errors against long double and those of
the same rows multiplied in double, over stretched shapes, axis-aligned plates
and tilted ones, with a layup that couples membrane and bending.  Bound as for
the homogeneous elements: the mean error of nine energies and of K_ij against
sqrt(K_ii K_jj), and here the worst of the latter, is at most sqrt(2) times the
double arithmetic's."""
import ctypes

import numpy as np
import pytest

from flexshell import _abi
from flexshell._lib import ptr
import test_fixed_quads as Q
import test_fixed_stretched as T
from test_fixed_stretched import lib  # noqa: F401


def layup(t):
    """A layup of thickness t, anisotropic, at an angle."""
    B = np.array([[1.0, 0, 0], [0.3, 0.4, 0], [-0.1, 0.15, 0.3]])
    Q = 1e11 * B @ B.T
    g = _abi.fs_layup_group()
    for f, M in (("A", t * Q), ("B", 0.1 * t ** 2 * Q), ("D", t ** 3 / 12 * Q), ("H", t * np.array([[5e9, 1e9], [1e9, 3e9]]))):
        getattr(g, f)[:] = list(np.asarray(M).flatten(order="F"))
    c, s = np.cos(0.4), np.sin(0.4)
    g.csmat[:] = list(np.array([[c, -s, 0], [s, c, 0], [0, 0, 1.0]]).flatten(order="F"))
    g.thickness = t
    return g


def run(lib, nen, avgk, X, N, t):  # noqa: F811
    n, nd = len(X), 6 * nen
    p = _abi.make_params(np.eye(3), np.eye(2), 0.0, 0.0, quads=nen == 4, transv_shear_formulation=avgk,
                         drilling_stiffness_scale=1.0)
    K, F, D = (np.zeros((n, nd, nd)) for _ in range(3))
    g = layup(t)
    a = [np.ascontiguousarray(v) for v in (X, N)]
    assert lib.stretched_layered(nen, avgk, ctypes.c_int64(n), *[ptr(v) for v in a], ctypes.byref(g), ctypes.byref(p),
                                 ptr(K), ptr(F), ptr(D)) == 0
    return K, F, D


def ratios(K, F, D, modes):
    s = np.sqrt(np.maximum(np.einsum("eii->ei", K), 0.0))
    s = s[:, :, None] * s[:, None, :]
    s[s == 0] = np.inf
    tiny = 1e-18
    r = [np.log((np.abs(F / s).max(axis=(1, 2)) + tiny) / (np.abs(D / s).max(axis=(1, 2)) + tiny)).mean(),
         np.log(np.abs(F / s).max() / np.abs(D / s).max())]
    for u in modes:
        en = np.einsum("ei,eij,ej->e", u, K, u)
        f, d = (np.abs(np.einsum("ei,eij,ej->e", u, E, u) / en) + tiny for E in (F, D))
        r.append(np.log(f / d).mean())
    return np.exp(r)


@pytest.mark.parametrize("flat", [True, False])
@pytest.mark.parametrize("avgk", [0, 1])
@pytest.mark.parametrize("lo", [1.0, 8.0, 64.0, 512.0])
def test_triangles(lib, lo, avgk, flat):  # noqa: F811
    X, R, N, _ = T.triangles(500, lo, 2 * lo, flat, int(lo))
    K, F, D = run(lib, 3, avgk, X, N, 0.01)
    r = ratios(K, F, D, T.modes(X, R))
    assert (r <= 2 ** 0.5).all(), r


@pytest.mark.parametrize("flat", [True, False])
@pytest.mark.parametrize("kind", ["square", "stretched16", "stretched64", "tapered", "sheared", "corner"])
def test_quads(lib, kind, flat):  # noqa: F811
    X, R, N, _ = Q.quads(kind, 500, flat, 4)
    K, F, D = run(lib, 4, 0, X, N, 0.01)
    r = ratios(K, F, D, Q.modes(X, R))
    assert (r <= 2 ** 0.5).all(), r
