"""The two host copies of a matrix: 1-based 64-bit and 0-based 32-bit indices."""
import ctypes

import numpy as np
import pytest

import flexshell as F
from flexshell import _abi
from flexshell._lib import FlexShellError, ptr

import problems as PB

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("assembler", [_abi.FS_ASM_SPARSE, _abi.FS_ASM_SPARSE_SYMM, _abi.FS_ASM_DIAG])
@pytest.mark.parametrize("n,free", [(1, False), (6, True), (6, False), (6, None)])
def test_the_same_matrix(assembler, n, free):
    xyz, conn, dof, nfree = PB.jittered_plate(n, False, wavy=0.0, seed=2)
    nrows = {True: nfree, False: dof.size, None: 0}[free]       # None: no rows at all
    femm = F.FEMMShellT3FF(conn, 0.01, F.materials.MatDeforElastIso(200e9, 0.3, 7850.0))
    geom0 = F.NodalField(xyz)
    dchi = F.NodalField(np.zeros((len(xyz), 6)))
    dchi.dofnums = np.asfortranarray(dof)
    with pytest.raises(FlexShellError) as ei:
        femm.ctx.call("fs_matrix_copy_i32", None, None, None)
    assert ei.value.code == _abi.FS_ERR_STATE
    femm.associategeometry(geom0)
    femm._sync_inputs(geom0, dchi)
    nnz = ctypes.c_int64()
    femm.ctx.call("fs_stiffness", F.FS_FP64, assembler, nrows, ctypes.byref(nnz))
    z = nnz.value
    c64, r64, v64 = np.zeros(nrows + 1, np.int64), np.zeros(z, np.int64), np.zeros(z)
    femm.ctx.call("fs_matrix_copy", ptr(c64), ptr(r64), ptr(v64))
    v32, r32, c32 = femm.ctx.matrix(nrows, z)
    assert r32.dtype == c32.dtype == np.int32
    assert np.array_equal(c32, c64 - 1) and np.array_equal(r32, r64 - 1) and np.array_equal(v32, v64)
    v = np.zeros(z)
    femm.ctx.call("fs_matrix_copy_i32", None, None, ptr(v))
    assert np.array_equal(v, v64)
    femm.close()
