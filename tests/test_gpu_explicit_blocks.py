"""The explicit step on node blocks at the edges of its launches: mesh sizes
around the lines between its forms (128 and 512 threads an SM), runs around a
captured graph's 64 steps, a matrix that is not symmetric, and a dof that no
node has; against the same loop in scipy."""
import ctypes

import numpy as np
import pytest

import flexshell as F
from flexshell import mesh
from flexshell._lib import ptr

pytestmark = pytest.mark.gpu

# of the largest value, after under a hundred steps: double differs in the order of
# rounding; float values and sums; float pairs
TOL = {F.FS_FP64: 1e-10, F.FS_MIXED: 2e-4, F.FS_MIXED_COMP: 1e-7}


def _plate(n, first_dof=1):
    xyz, quad = mesh.jittered_plate_q(n, 1.0, 0.15, 3, None)
    fixed = np.zeros((len(xyz), 6), bool)
    fixed[xyz[:, 0] < 1e-9] = True
    dof, nfree = mesh.numberdofs(fixed)
    dof = np.asfortranarray(dof + (first_dof - 1))
    femm = F.FEMMShellQ4RS(quad, 0.01, F.materials.MatDeforElastIso(200e9, 0.3, 7850.0))
    geom0 = F.NodalField(xyz)
    dchi = F.NodalField(np.zeros((len(xyz), 6)))
    dchi.dofnums = dof
    femm.associategeometry(geom0)
    n = nfree + first_dof - 1
    K = femm.stiffness(F.SysmatAssemblerFFBlock(n), geom0, None, None, dchi).tocsr()
    return femm, K, n


def _vectors(n, K):
    rng = np.random.default_rng(1)
    m = abs(K).sum(axis=1).A1 if hasattr(abs(K).sum(axis=1), "A1") else np.asarray(abs(K).sum(axis=1)).ravel()
    m = np.where(m > 0, m, 1.0)     # 2 / omega of this mass is above 1.4
    C = 0.01 * m
    return m, C, rng.normal(0, 1e-3, n)


def _reference(K, m, C, dt, V, steps):
    U, A = np.zeros_like(V), np.zeros_like(V)
    V = V.copy()
    inv = 1.0 / (m + dt / 2 * C)
    for _ in range(steps):
        U = U + dt * V + dt * dt / 2 * A
        f = -(K @ U) - C * (V + dt / 2 * A)
        V = V + dt / 2 * A
        A = inv * f
        V = V + dt / 2 * A
    return U, V, A


def _check(femm, K, m, C, V0, precision, runs, dt=1.0):
    n = len(m)
    ref = _reference(K, m, C, dt, V0, sum(runs))
    inv = np.ascontiguousarray(1.0 / (m + dt / 2 * C))
    z = np.zeros(n)
    call = femm.ctx.call
    call("fs_explicit_setup", precision, ptr(inv), ptr(C), ctypes.c_double(dt))
    out = []
    for parts in (runs, [sum(runs)]):      # in parts and at once: the same bits
        call("fs_explicit_set_state", ptr(z), ptr(V0), ptr(z))
        for k in parts:
            call("fs_explicit_run", k)
        got = [np.zeros(n) for _ in range(3)]
        call("fs_explicit_get_state", *[ptr(g) for g in got])
        out.append(got)
    for a, b, r in zip(out[0], out[1], ref):
        assert np.array_equal(a, b)
        assert np.abs(a - r).max() <= TOL[precision] * np.abs(r).max()


@pytest.mark.parametrize("precision", [F.FS_FP64, F.FS_MIXED, F.FS_MIXED_COMP])
@pytest.mark.parametrize("n", [1, 2, 79, 80, 160, 161])
def test_sizes_and_runs(n, precision):
    femm, K, nd = _plate(n)
    m, C, V0 = _vectors(nd, K)
    _check(femm, K, m, C, V0, precision, [1, 64, 2] if n < 100 else [3, 65])
    femm.close()


@pytest.mark.parametrize("precision", [F.FS_FP64, F.FS_MIXED, F.FS_MIXED_COMP])
def test_unsymmetric_values(precision):
    import torch
    femm, K, nd = _plate(7)
    rp, ci, v = ctypes.c_void_p(), ctypes.c_void_p(), ctypes.c_void_p()
    n, nnz = ctypes.c_int64(), ctypes.c_int64()
    femm.ctx.call("fs_matrix_device", ctypes.byref(rp), ctypes.byref(ci), ctypes.byref(v), ctypes.byref(n),
                  ctypes.byref(nnz))

    class View:
        __cuda_array_interface__ = {"shape": (nnz.value,), "typestr": "<f8", "data": (v.value, False), "version": 3}

    vals = torch.as_tensor(View(), device="cuda")
    vals *= 1.0 + 0.1 * torch.rand(nnz.value, dtype=torch.float64, device="cuda",
                                   generator=torch.Generator("cuda").manual_seed(5))
    torch.cuda.synchronize()
    K = K.copy()
    K.data = vals.cpu().numpy()
    m, C, V0 = _vectors(nd, K)
    _check(femm, K, m, C, V0, precision, [5, 20], dt=0.3)
    femm.close()


def test_a_dof_without_a_node():
    femm, K, nd = _plate(5, first_dof=3)   # dofs 1 and 2: empty rows that keep moving
    assert K[:2].nnz == 0
    m, C, V0 = _vectors(nd, K)
    C[:2] = 0.0
    _check(femm, K, m, C, V0, F.FS_FP64, [1, 3, 65])
    femm.close()
