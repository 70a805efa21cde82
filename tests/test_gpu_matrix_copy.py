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


def test_large_copies_into_any_memory():
    # results of a megabyte and more: into new pages, used ones, and an address
    # inside a page, with what lies around them untouched
    xyz, conn, dof, nfree = PB.jittered_plate(60, False, wavy=0.02, seed=2)
    femm = F.FEMMShellT3FF(conn, 0.01, F.materials.MatDeforElastIso(200e9, 0.3, 7850.0))
    geom0 = F.NodalField(xyz)
    dchi = F.NodalField(np.zeros((len(xyz), 6)))
    dchi.dofnums = np.asfortranarray(dof)
    femm.associategeometry(geom0)
    K = femm.stiffness(F.SysmatAssemblerSparse(), geom0, None, None, dchi)
    z = K.nnz
    assert 8 * z > 1 << 20
    for shift in (0, 1, 511):
        for fill in (None, -7.0):
            buf = np.empty(z + 1024) if fill is None else np.full(z + 1024, fill)
            buf[:shift], buf[shift + z:] = 3.0, 4.0
            femm.ctx.call("fs_matrix_copy_i32", None, None, ptr(buf[shift:]))
            assert np.array_equal(buf[shift:shift + z], K.data)
            assert (buf[:shift] == 3.0).all() and (buf[shift + z:] == 4.0).all()
    femm.close()
