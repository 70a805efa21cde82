"""FS_FP64 element matrices on the GPU where a whole group of the fixed point's
numbers is zero: zero thickness, alone and among others, and materials without
membrane and bending or without transverse shear stiffness.  The zero-dropping
assembler's kernels (double) and the host's double arithmetic are the reference;
tolerance 1e-12 of the largest entry, the FP64 parity bound."""
import numpy as np
import pytest

import flexshell as F
from test_fixed_elements import _elements, lib  # noqa: F401
from test_fixed_groups import KINDS, fixed_and_double, material

pytestmark = pytest.mark.gpu


class _Moduli:
    """A material whose plane-stress and shear stiffness are those of `material`."""

    def __init__(self, kind):
        self.D = np.eye(6)
        Dps, Dt = material(kind)
        ix = np.ix_([0, 1, 3], [0, 1, 3])
        self.D[ix] = Dps
        self.D[np.ix_([4, 5], [4, 5])] = np.diag(np.diag(Dt))

    def tangentmoduli(self):
        return self.D

    def massdensity(self):
        return 1.0


def _femm(nen, X, N, valid, t, kind):
    n = len(X)
    conn = np.arange(1, n * nen + 1, dtype=np.int64).reshape(n, nen)
    femm = (F.FEMMShellT3FF if nen == 3 else F.FEMMShellQ4RS)(conn, t, _Moduli(kind))
    geom0 = F.NodalField(X.reshape(-1, 3))
    femm._upload_mesh(geom0)
    femm.set_normals(N.reshape(-1, 3), valid.reshape(-1))
    dchi = F.NodalField(np.zeros((n * nen, 6)))
    dchi.numberdofs()
    return femm, geom0, dchi


@pytest.mark.parametrize("nen", [3, 4])
@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("flat", [False, True])
def test_vanishing_stiffness(lib, nen, kind, flat):  # noqa: F811
    X, N, valid, t = _elements(nen, 70, 21, flat=flat, size=(-2, 1))
    Dps, Dt = material(kind)
    _, D, _ = fixed_and_double(lib, nen, X, N, valid, t, Dps, np.diag(np.diag(Dt)))
    femm, geom0, dchi = _femm(nen, X, N, valid, t, kind)
    G = femm.element_matrices(geom0)
    mx = np.abs(D).max(axis=(1, 2))
    assert (np.abs(G - D).max(axis=(1, 2)) <= 1e-12 * mx).all()
    femm.close()


@pytest.mark.parametrize("nen", [3, 4])
@pytest.mark.parametrize("every", [1, 3])
def test_zero_thickness(lib, nen, every):  # noqa: F811
    X, N, valid, t = _elements(nen, 70, 22, size=(-2, 1))
    t[::every] = 0.0
    femm, geom0, dchi = _femm(nen, X, N, valid, t, "iso")
    G = femm.element_matrices(geom0)
    assert (G[::every] == 0).all()
    assert every == 1 or (np.abs(G[1::3]).max(axis=(1, 2)) > 0).all()
    K = femm.stiffness(F.SysmatAssemblerSparse(), geom0, None, None, dchi)
    S = femm.stiffness(F.SysmatAssemblerSparseSymm(), geom0, None, None, dchi)
    mx = np.abs(G).max()
    assert abs(K - S).max() <= 1e-12 * mx
    femm.close()
