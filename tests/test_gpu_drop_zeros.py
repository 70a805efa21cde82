"""The assembler that drops exact zeros against the one that keeps them, entry by
entry, over one context's changing matrices (its buffers change places)."""
import numpy as np
import pytest

import flexshell as F

import problems as PB

pytestmark = pytest.mark.gpu


def _same(A, B):
    A, B = A.tocsr(), B.tocsr()
    assert np.array_equal(A.indptr, B.indptr) and np.array_equal(A.indices, B.indices)
    assert np.array_equal(A.data, B.data)


def _kept(K):
    K = K.tocsr().copy()
    K.eliminate_zeros()
    return K


@pytest.mark.parametrize("n", [12, 13, 294, 296])
def test_row_counts_around_the_scans_forms(n):
    # the row lengths are summed in chunks of 1,024 rows: one chunk and two, and on
    # either side of 512 chunks (6 dofs a node, (n + 1)^2 nodes)
    xyz, conn, dof, nfree = PB.jittered_plate(n, True, wavy=0.0, seed=1)
    femm = F.FEMMShellQ4RS(conn, 0.01, F.materials.MatDeforElastIso(200e9, 0.3, 7850.0))
    geom0 = F.NodalField(xyz)
    dchi = F.NodalField(np.zeros((len(xyz), 6)))
    dchi.numberdofs()
    femm.associategeometry(geom0)
    A = femm.stiffness(F.SysmatAssemblerSparse(), geom0, None, None, dchi, precision=F.FS_MIXED)
    B = femm.stiffness(F.SysmatAssemblerSparseSymm(), geom0, None, None, dchi, precision=F.FS_MIXED)
    _same(_kept(A), B)
    femm.close()


@pytest.mark.parametrize("quads", [False, True])
@pytest.mark.parametrize("n", [1, 2, 5, 17, 40])
@pytest.mark.parametrize("wavy", [0.0, 0.03])
def test_entries(quads, n, wavy):
    # float values: both assemblers run the same element kernels
    xyz, conn, dof, nfree = PB.jittered_plate(n, quads, wavy=wavy, seed=n)
    cls = F.FEMMShellQ4RS if quads else F.FEMMShellT3FF
    femm = cls(conn, 0.01, F.materials.MatDeforElastIso(200e9, 0.3, 7850.0))
    geom0 = F.NodalField(xyz)
    dchi = F.NodalField(np.zeros((len(xyz), 6)))
    dchi.dofnums = np.asfortranarray(dof)
    femm.associategeometry(geom0)
    full = [F.SysmatAssemblerSparse(), F.SysmatAssemblerFFBlock(F.SysmatAssemblerSparse(), nfree)]
    drop = [F.SysmatAssemblerSparseSymm(), F.SysmatAssemblerFFBlock(F.SysmatAssemblerSparseSymm(), nfree)]
    for precision in (F.FS_MIXED, F.FS_MIXED_COMP):
        for k in (0, 1, 0):              # all dofs, the free ones (rows of any length), all again
            A = femm.stiffness(full[k], geom0, None, None, dchi, precision=precision)
            for _ in range(2):
                B = femm.stiffness(drop[k], geom0, None, None, dchi, precision=precision)
                _same(_kept(A), B)
            assert wavy or B.nnz < A.nnz
            _same(A, femm.stiffness(full[k], geom0, None, None, dchi, precision=precision))
    M = femm.mass(F.SysmatAssemblerSparseDiag(), geom0, dchi)
    _same(_kept(M), femm.mass(F.SysmatAssemblerSparseSymm(), geom0, dchi))
    femm.close()
