"""FS_FP64 element matrices on the GPU at the edges of their kernels: element
counts around a group of 32, and degenerate elements, which leave the fixed
point for the double kernel, among good ones."""
import numpy as np
import pytest

import flexshell as F
from flexshell import _abi
from flexshell._lib import FlexShellError
from test_fixed_elements import _elements, _run, lib  # noqa: F401

pytestmark = pytest.mark.gpu

STEEL = dict(E=2.0e11, nu=0.3, rho=7850.0)


def _femm(nen, X, N, valid, t):
    """One mesh of separate elements."""
    n = len(X)
    conn = np.arange(1, n * nen + 1, dtype=np.int64).reshape(n, nen)
    cls = F.FEMMShellT3FF if nen == 3 else F.FEMMShellQ4RS
    femm = cls(conn, t, F.materials.MatDeforElastIso(STEEL["E"], STEEL["nu"], STEEL["rho"]))
    geom0 = F.NodalField(X.reshape(-1, 3))
    femm._upload_mesh(geom0)
    femm.set_normals(N.reshape(-1, 3), valid.reshape(-1))
    return femm, geom0


@pytest.mark.parametrize("nen", [3, 4])
@pytest.mark.parametrize("n", [1, 31, 32, 33, 65, 127])
def test_against_the_host_build(lib, nen, n):  # noqa: F811
    # the same arithmetic but for contraction: within the FP64 parity bound
    X, N, valid, t = _elements(nen, n, n, tilt=0.3, warp=0.02 * (nen == 4), size=(-2, 1))
    K, D, ok = _run(lib, nen, X, N, valid, t)
    assert ok.all()
    femm, geom0 = _femm(nen, X, N, valid, t)
    G = femm.element_matrices(geom0)
    mx = np.abs(D).max(axis=(1, 2))
    assert (np.abs(G - D).max(axis=(1, 2)) <= 1e-12 * mx).all()
    assert (np.abs(G - K).max(axis=(1, 2)) <= 1e-12 * mx).all()
    femm.close()


def test_degenerate_triangles_among_good_ones(lib):  # noqa: F811
    n = 70
    X, N, valid, t = _elements(3, n, 5, size=(-1, 0))
    femm, geom0 = _femm(3, X, N, valid, t)
    good = femm.element_matrices(geom0)
    femm.close()
    Y = X.copy()
    bad = np.array([0, 33, 69])
    # exactly degenerate (any other way of drawing them leaves a rounding error
    # of an area, and a finite matrix)
    Y[bad[0], 1] = Y[bad[0], 0]                                   # the first two nodes in one place
    Y[bad[1]] = np.arange(3.0)[:, None] * [1.0, 0.0, 0.0]         # nodes on an axis
    Y[bad[2]] *= 1e-90                                            # next to a double's limits
    femm, geom0 = _femm(3, Y, N, valid, t)
    G = femm.element_matrices(geom0)
    rest = np.setdiff1d(np.arange(n), bad)
    assert np.array_equal(G[rest], good[rest])
    _, D, ok = _run(lib, 3, Y, N, valid, t)
    assert not ok[bad].any() and ok[rest].all()
    for e in bad[:2]:
        assert not np.isfinite(G[e]).all()
        assert np.array_equal(np.isfinite(G[e]), np.isfinite(D[e]))
    if np.isfinite(D[bad[2]]).all():
        assert np.abs(G[bad[2]] - D[bad[2]]).max() <= 1e-12 * np.abs(D[bad[2]]).max()
    # assembled: the good elements' values are there, through the second gather
    dchi = F.NodalField(np.zeros((Y.size // 3, 6)))
    dchi.numberdofs()
    Ka = femm.stiffness(F.SysmatAssemblerSparse(), geom0, None, None, dchi).tocsr()
    for e in rest[:5]:
        d = np.arange(18 * e, 18 * e + 18)
        assert np.array_equal(Ka[d][:, d].toarray(), G[e])
    femm.close()


def test_singular_quadrilateral_is_an_error():
    X, N, valid, t = _elements(4, 40, 6, size=(-1, 0))
    X[37] = [0.5, 0.25, 0.0]   # one point four times: zero tangents (the determinant is zero exactly)
    femm, geom0 = _femm(4, X, N, valid, t)
    with pytest.raises(FlexShellError) as ei:
        femm.element_matrices(geom0)
    assert ei.value.code == _abi.FS_ERR_SINGULAR_METRIC
    femm.close()


def test_dropping_zeros_keeps_the_smallest_entries():
    # one triangle tilted by a rounding error: in double its drilling rows hold
    # entries of relative size 1e-25, which are not zeros
    X = np.array([[0.0, 0.0, 0.0], [1.0, 0.1, 1e-16], [0.2, 0.9, 0.0]])
    femm = F.FEMMShellT3FF(np.array([[1, 2, 3]]), 0.01, F.materials.MatDeforElastIso(STEEL["E"], STEEL["nu"], STEEL["rho"]))
    geom0 = F.NodalField(X)
    dchi = F.NodalField(np.zeros((3, 6)))
    dchi.numberdofs()
    femm.associategeometry(geom0)
    K = femm.stiffness(F.SysmatAssemblerSparseSymm(), geom0, None, None, dchi).tocsr()
    assert K[5::6].nnz > 0 and (K.data != 0).all()
    femm.close()
