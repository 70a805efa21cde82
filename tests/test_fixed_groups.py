"""Groups of the FS_FP64 elements' fixed point whose numbers are all zero
(csrc/fs_elem_fixed.cuh on the host): elements of zero thickness, and materials
without membrane and bending or without transverse shear stiffness, against the
same elements in double.

Tolerance: 1e-12 of the largest entry, the repository's FP64 parity bound; a
matrix that is exactly zero in double is exactly zero."""
import ctypes

import numpy as np
import pytest

from flexshell import _abi, materials
from flexshell._lib import ptr
from test_fixed_elements import _elements, lib  # noqa: F401


def fixed_and_double(lib, nen, X, N, valid, t, Dps, Dt):  # noqa: F811
    n, nd = len(X), 6 * nen
    p = _abi.make_params(Dps, Dt, 7850.0, 0.0, quads=nen == 4, drilling_stiffness_scale=1.0)
    K, D, ok = np.zeros((n, nd, nd)), np.zeros((n, nd, nd)), np.zeros(n, np.uint8)
    a = [np.ascontiguousarray(v) for v in (X, N, valid, t)]
    assert lib.fixed_elements(nen, ctypes.c_int64(n), *[ptr(v) for v in a], ctypes.byref(p), ptr(K), ptr(D), ptr(ok)) == 0
    return K, D, ok.astype(bool)


def material(kind):
    """Plane-stress and transverse-shear stiffness, of unit size."""
    Dps, Dt = materials.shell_material_stiffness(materials.MatDeforElastIso(1.0, 0.3, 1.0))
    if kind == "no shear":
        Dt = 0.0 * Dt
    elif kind == "one shear":
        Dt = np.diag([1.0, 0.0])
    elif kind == "no plane":
        Dps = 0.0 * Dps
    elif kind == "one way":
        Dps = np.diag([1.0, 0.0, 0.0])
    elif kind == "full":
        B = np.array([[1.0, 0, 0], [0.4, 0.7, 0], [-0.3, 0.2, 0.5]])
        Dps, Dt = B @ B.T, np.array([[0.5, 0.1], [0.1, 0.02]])
    return Dps, Dt


KINDS = ["iso", "no shear", "one shear", "no plane", "one way", "full"]


@pytest.mark.parametrize("nen", [3, 4])
@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("flat", [False, True])
def test_vanishing_stiffness(lib, nen, kind, flat):  # noqa: F811
    X, N, valid, t = _elements(nen, 60, 11, flat=flat, warp=0.02 * (nen == 4 and not flat))
    K, D, ok = fixed_and_double(lib, nen, X, N, valid, t, *material(kind))
    assert ok.all()
    mx = np.abs(D).max(axis=(1, 2))
    assert (np.abs(K - D).max(axis=(1, 2)) <= 1e-12 * mx).all()


@pytest.mark.parametrize("nen", [3, 4])
@pytest.mark.parametrize("flat", [False, True])
def test_zero_thickness(lib, nen, flat):  # noqa: F811
    X, N, valid, t = _elements(nen, 60, 12, flat=flat)
    t[::3] = 0.0
    K, D, ok = fixed_and_double(lib, nen, X, N, valid, t, *material("iso"))
    assert ok.all()
    assert (D[::3] == 0).all() and (K[::3] == 0).all()
    mx = np.abs(D).max(axis=(1, 2))
    assert (np.abs(K - D).max(axis=(1, 2)) <= 1e-12 * mx).all()
