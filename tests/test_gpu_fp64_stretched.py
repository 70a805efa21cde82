"""FS_FP64 on the GPU with triangles that are too long for the fixed point: they get
the double kernel's matrices to the bit (those of the assembler that drops zeros,
which runs that kernel alone), by each way to a stiffness, and the others beside
them keep theirs."""

import numpy as np
import pytest

import flexshell as F
from test_fixed_stretched import triangles

pytestmark = pytest.mark.gpu


def _femm(X, N, t):
    n = len(X)
    conn = np.arange(1, 3 * n + 1, dtype=np.int64).reshape(n, 3)
    femm = F.FEMMShellT3FF(conn, t, F.materials.MatDeforElastIso(2.0e11, 0.3, 7850.0))
    geom0 = F.NodalField(X.reshape(-1, 3))
    femm._upload_mesh(geom0)
    femm.set_normals(N.reshape(-1, 3), np.ones(3 * n, bool))
    dchi = F.NodalField(np.zeros((3 * n, 6)))
    dchi.numberdofs()
    return femm, geom0, dchi


def _blocks(K, n):
    K = K.tocsr()
    return np.array([K[18 * e:18 * e + 18, 18 * e:18 * e + 18].toarray() for e in range(n)])


@pytest.mark.parametrize("flat", [True, False])
@pytest.mark.parametrize("which", [slice(None), slice(0, 0), slice(5, None, 7)])
def test_long_triangles_are_the_double_kernels(flat, which):
    n = 97
    a, b = triangles(n, 1.0, 30.0, flat, 1), triangles(n, 40.0, 400.0, flat, 2)
    X, N, t = (v.copy() for v in (a[0], a[2], a[3]))
    for v, w in zip((X, N, t), (b[0], b[2], b[3])):
        v[which] = w[which]
    far = np.zeros(n, bool)
    far[which] = True
    femm, geom0, dchi = _femm(X, N, t)
    double = _blocks(femm.stiffness(F.SysmatAssemblerSparseSymm(), geom0, None, None, dchi), n)
    got = _blocks(femm.stiffness(F.SysmatAssemblerSparse(), geom0, None, None, dchi), n)
    assert np.array_equal(got[far], double[far])
    if not far.all():
        assert not np.array_equal(got[~far], double[~far])
    mx = np.abs(double).max(axis=(1, 2))
    assert (np.abs(got - double).max(axis=(1, 2)) <= 1e-12 * mx).all()
    assert np.array_equal(femm.element_matrices(geom0), got)
    # with nothing but the long ones changed, the others stay as they are
    Y = X.copy()
    Y[far] = triangles(n, 40.0, 400.0, flat, 3)[0][far]
    femm2, geom2, dchi2 = _femm(Y, N, t)
    again = femm2.element_matrices(geom2)
    assert np.array_equal(again[~far], got[~far])
    femm.close()
    femm2.close()
