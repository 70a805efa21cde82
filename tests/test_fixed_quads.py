"""Accuracy of the FS_FP64 elements on quadrilaterals: the fixed point
(csrc/fs_elem_fixed.cuh) and the double arithmetic that it stands for, both
against the same element in long double, over stretched, tapered and sheared
shapes, axis-aligned plates and tilted ones.  Bound as for the triangles: the
mean error of nine energies and of K_ij against sqrt(K_ii K_jj) is at most
sqrt(2) times the double arithmetic's."""
import ctypes

import numpy as np
import pytest

from flexshell import _abi, materials
from flexshell._lib import ptr
from test_fixed_stretched import lib  # noqa: F401


def quads(kind, n, flat, seed):
    rng = np.random.default_rng(seed)
    P = np.zeros((n, 4, 2)) + [[0, 0], [1, 0], [1, 1], [0, 1.0]] + 0.1 * rng.uniform(-1, 1, (n, 4, 2))
    if kind.startswith("stretched"):
        P[:, :, 0] *= float(kind[9:])
    elif kind == "tapered":
        P[:, 2, 0], P[:, 3, 0] = 0.5 + 0.05 * rng.uniform(0.1, 1, n), 0.5 - 0.05 * rng.uniform(0.1, 1, n)
    elif kind == "sheared":
        P[:, :, 0] += 2.0 * P[:, :, 1]
    elif kind == "corner":
        P[:, 2] = 0.5 + 0.06 * rng.uniform(0.5, 1, (n, 1))
    for e in range(n):
        P[e] = np.roll(P[e], rng.integers(4), axis=0)
    P *= 10.0 ** rng.uniform(-2, 0, n)[:, None, None]
    R = np.broadcast_to(np.eye(3), (n, 3, 3))
    if not flat:
        R, _ = np.linalg.qr(rng.normal(size=(n, 3, 3)))
        R = R * np.sign(np.linalg.det(R))[:, None, None]
    size = np.abs(P).max(axis=(1, 2))
    X = np.einsum("eai,eic->eac", P, R[:, :2])
    if not flat:
        X = X + 0.01 * size[:, None, None] * rng.uniform(-1, 1, (n, 4, 1)) * R[:, None, 2]
    N = np.repeat(R[:, None, 2], 4, axis=1) + (0.0 if flat else 0.03) * rng.uniform(-1, 1, (n, 4, 3))
    N /= np.linalg.norm(N, axis=2, keepdims=True)
    return X, R, N, size * 10.0 ** rng.uniform(-3, -1, n)


def modes(X, R):
    """Nine displacement fields at the nodes, in the element plane's axes."""
    x, y, _ = np.moveaxis(np.einsum("eac,eic->eai", X - X.mean(axis=1, keepdims=True), R), 2, 0)
    o, one = np.zeros_like(x), np.ones_like(x)
    local = [(x, o, o, o, o, o), (o, y, o, o, o, o), (y / 2, x / 2, o, o, o, o),
             (o, o, -x * x / 2, o, x, o), (o, o, -y * y / 2, -y, o, o), (o, o, -x * y, -x, y, o),
             (o, o, o, o, one, o), (o, o, o, one, o, o), (o, o, o, o, x, o)]
    u = np.array(local).transpose(0, 2, 3, 1)
    g = np.concatenate([np.einsum("meai,eic->meac", u[..., :3], R), np.einsum("meai,eic->meac", u[..., 3:], R)], axis=3)
    return g.reshape(9, len(X), 24)


@pytest.mark.parametrize("flat", [True, False])
@pytest.mark.parametrize("kind", ["square", "stretched4", "stretched16", "stretched64", "tapered", "sheared", "corner"])
def test_no_further_off_than_double(lib, kind, flat):  # noqa: F811
    n = 800
    X, R, N, t = quads(kind, n, flat, 4)
    Dps, Dt = materials.shell_material_stiffness(materials.MatDeforElastIso(2.0e11, 0.3, 7850.0))
    p = _abi.make_params(Dps, Dt, 7850.0, 0.0, quads=True, drilling_stiffness_scale=1.0)
    K, F, D = (np.zeros((n, 24, 24)) for _ in range(3))
    a = [np.ascontiguousarray(v) for v in (X, N, t)]
    assert lib.stretched_quads(ctypes.c_int64(n), *[ptr(v) for v in a], ctypes.byref(p), ptr(K), ptr(F), ptr(D)) == 0
    s = np.sqrt(np.maximum(np.einsum("eii->ei", K), 0.0))
    s = s[:, :, None] * s[:, None, :]
    s[s == 0] = np.inf
    tiny = 1e-18
    r = [np.log((np.abs(F / s).max(axis=(1, 2)) + tiny) / (np.abs(D / s).max(axis=(1, 2)) + tiny)).mean()]
    for u in modes(X, R):
        en = np.einsum("ei,eij,ej->e", u, K, u)
        f, d = (np.abs(np.einsum("ei,eij,ej->e", u, E, u) / en) + tiny for E in (F, D))
        r.append(np.log(f / d).mean())
    assert (np.exp(r) <= 2 ** 0.5).all(), np.exp(r)
