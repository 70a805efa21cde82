"""Performance cases of the shell and beam assembly and of the explicit step.

Each case is one piece of work that a program using this framework has it do,
called as such a program calls it: the Python classes with host results for
the small and ordinary analyses (kinds "call" and "model"), the C entry
points with the matrix left on the device for the large assemblies
("assembly", "panels", "beams") and the time-step loop ("explicit").

exact() restates the element formulas in dense double precision (torch) and
sums them into the same layout, without the library.
"""
import ctypes
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "finetoolsflexstructures.jl_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import flexshell as F  # noqa: E402
from flexshell import _abi  # noqa: E402
from flexshell._lib import Context, ptr  # noqa: E402

PRECISION = {"fp64": _abi.FS_FP64, "mixed": _abi.FS_MIXED, "comp": _abi.FS_MIXED_COMP}
ASSEMBLER = {"sparse": _abi.FS_ASM_SPARSE, "symm": _abi.FS_ASM_SPARSE_SYMM}
E, NU, RHO = 200e9, 0.3, 7850.0  # steel
STAB = {"t3": 5 / 12 / 1.5, "q4": 0.1}  # the FEMMs' default stab_fun coefficients


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def _assembly(el, layered, precision, nx, ny, wave, assembler="sparse", name=None):
    c = {"kind": "assembly", "el": el, "layered": layered, "precision": precision, "nx": nx, "ny": ny,
         "wave": wave, "assembler": assembler}
    return dict(c, name=name) if name else c


def _explicit(el, precision, n, steps, load, name=None):
    c = {"kind": "explicit", "el": el, "precision": precision, "n": n, "steps": steps, "load": load}
    return dict(c, name=name) if name else c


def listed():
    return [
        # the smallest call: configuration 1's plate through stiffness() with its
        # defaults (FP64, SysmatAssemblerSparseSymm), as in a static analysis or a test
        {"name": "t3_call_32", "kind": "call", "el": "t3", "nx": 32, "ny": 32},
        # a whole small model from its mesh: associategeometry!, lumped mass and
        # free-free stiffness, what a modal analysis asks before its eigensolver
        {"name": "q4_model_120x75", "kind": "model", "el": "q4", "nx": 120, "ny": 75},
        # an ordinary flat plate in the default precision and with the default
        # assembler (the exact zeros of its uncoupled dofs are dropped)
        _assembly("t3", False, "fp64", 300, 211, False, "symm", "t3_fp64_flat_300x211"),
        # the benchmark's plate in its headline precision
        _assembly("t3", False, "comp", 1024, 1024, True, "sparse", "t3_comp_1024"),
        # the benchmark's other element in the default precision
        _assembly("q4", False, "fp64", 512, 512, True, "sparse", "q4_fp64_512"),
        # quads in the compensated precision, a ragged size
        _assembly("q4", False, "comp", 333, 401, True, "sparse", "q4_comp_333x401"),
        # the layered plate of configuration 4
        _assembly("q4", True, "comp", 512, 512, False, "sparse", "q4layer_comp_512"),
        # layered triangles, two layup groups, default precision
        _assembly("t3", True, "fp64", 257, 190, True, "sparse", "t3layer_fp64_257x190"),
        # configuration 3: 64 uneven cylindrical panels assembled together
        {"name": "panels_mixed_64", "kind": "panels", "precision": "mixed", "panels": 64, "nmax": 256},
        # the reference's published explicit plate (51,200 triangles), with its load
        _explicit("t3", "fp64", 160, 640, True, "explicit_t3_fp64_160"),
        # configuration 5's plate in the compensated precision, 320 steps between two looks
        _explicit("q4", "comp", 512, 320, False, "explicit_q4_comp_512"),
        # a beam lattice in a deformed state: one stiffness of a Newton iteration
        {"name": "beams_60", "kind": "beams", "n": 60, "timoshenko": False},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["call", "model", "assembly", "assembly", "assembly", "assembly", "panels", "explicit",
                       "explicit", "beams"])
    el = rng.choice(["t3", "q4"])
    if kind in ("call", "model"):
        return {"kind": kind, "el": el, "nx": _log_int(rng, 5, 120), "ny": _log_int(rng, 5, 75)}
    if kind == "assembly":
        precision = rng.choice(["fp64", "mixed", "comp"])
        layered = rng.random() < 0.3
        hi = 1000 if el == "t3" and not layered else 500
        # the layered plates keep their explicit zeros: which of their entries cancel
        # to an exact zero is a matter of rounding
        return _assembly(el, layered, precision, _log_int(rng, 9, hi), _log_int(rng, 9, hi), rng.random() < 0.7,
                         "sparse" if layered else rng.choice(["sparse", "symm"]))
    if kind == "panels":
        return {"kind": kind, "precision": rng.choice(["fp64", "mixed", "comp"]), "panels": rng.randint(4, 64),
                "nmax": _log_int(rng, 24, 200)}
    if kind == "explicit":
        return _explicit(el, rng.choice(["fp64", "mixed", "comp"]), _log_int(rng, 12, 400), rng.randint(50, 300),
                         rng.random() < 0.5)
    return {"kind": "beams", "n": _log_int(rng, 4, 60), "timoshenko": rng.random() < 0.5}


# ---------------------------------------------------------------------------
# inputs (host arrays made from the seed alone)
# ---------------------------------------------------------------------------
def _plate(el, nx, ny, seed, wave, jitter=0.2):
    """A jittered nx x ny plate on [0,1]^2, flat or with z = a sin(pi x) sin(pi y):
    coordinates, 1-based connectivity."""
    rng = np.random.Generator(np.random.PCG64(seed))
    X, Y = np.meshgrid(np.linspace(0, 1, nx + 1), np.linspace(0, 1, ny + 1))
    xyz = np.zeros(((nx + 1) * (ny + 1), 3), order="F")
    inner = np.zeros((ny + 1, nx + 1), bool)
    inner[1:-1, 1:-1] = True
    d = rng.uniform(-jitter, jitter, size=(2, ny + 1, nx + 1)) * inner
    xyz[:, 0] = (X + d[0] / nx).ravel()
    xyz[:, 1] = (Y + d[1] / ny).ravel()
    if wave:
        xyz[:, 2] = rng.uniform(0.008, 0.012) * np.sin(np.pi * xyz[:, 0]) * np.sin(np.pi * xyz[:, 1])
    i = np.repeat(np.arange(1, nx + 1), ny)
    j = np.tile(np.arange(ny), nx)
    f = j * (nx + 1) + i
    quad = np.stack([f, f + 1, f + nx + 2, f + nx + 1], axis=1).astype(np.int64)
    if el == "q4":
        return xyz, quad
    tri = np.empty((2 * len(quad), 3), dtype=np.int64)
    tri[0::2] = quad[:, [0, 1, 3]]
    tri[1::2] = quad[:, [1, 2, 3]]
    return xyz, tri


def _number(fixed):
    """numberdofs!: free dofs first, node by node; the fixed ones after them."""
    free = ~fixed.ravel()
    dof = np.empty(free.size, dtype=np.int64)
    nfree = int(free.sum())
    dof[free] = np.arange(1, nfree + 1)
    dof[~free] = np.arange(nfree + 1, free.size + 1)
    return np.asfortranarray(dof.reshape(fixed.shape)), nfree


def _edge(xyz):
    x, y = xyz[:, 0], xyz[:, 1]
    return (x < 1e-9) | (x > 1 - 1e-9) | (y < 1e-9) | (y > 1 - 1e-9)


def _layup():
    """Ply stiffness (orthotropic, plane stress) of configuration 4's lamina and
    the two layups used: [0/90/90/0] and [30/-30]."""
    E1, E2, nu12, G12, G13, G23 = 140e9, 10e9, 0.3, 5e9, 5e9, 3.5e9
    nu21 = nu12 * E2 / E1
    d = 1 - nu12 * nu21
    Dps = np.array([[E1 / d, nu12 * E2 / d, 0], [nu12 * E2 / d, E2 / d, 0], [0, 0, G12]])
    Dts = np.diag([G13, G23])
    return Dps, Dts, 1600.0, 0.25e-3, [(0, 90, 90, 0), (30, -30)]


def _panels(case, seed):
    """Cylindrical panels (R 25, L 50, 80 degrees), n x n quads in triangles."""
    rng = np.random.Generator(np.random.PCG64(seed))
    sizes = np.random.Generator(np.random.PCG64(3))  # the same work for every seed
    out = []
    for _ in range(case["panels"]):
        n = int(sizes.integers(16, case["nmax"] + 1))
        xyz, conn = _plate("t3", n, n, int(rng.integers(1 << 30)), False, jitter=0.05)
        a = xyz[:, 0] * (80 / 180 * np.pi)
        p = np.asfortranarray(np.stack([25 * np.sin(a), 50 * xyz[:, 1], 25 * (np.cos(a) - 1)], 1))
        out.append((p, conn, float(rng.uniform(0.1, 0.5))))
    return out


def _beams(case, seed):
    """An n^3 lattice of beams with random sections, displacements and rotations."""
    n = case["n"]
    rng = np.random.Generator(np.random.PCG64(seed))
    g = np.arange(n, dtype=np.float64)
    xyz = np.stack(np.meshgrid(g, g, g, indexing="ij"), -1).reshape(-1, 3) + rng.uniform(-0.1, 0.1, (n ** 3, 3))
    idx = np.arange(1, n ** 3 + 1).reshape(n, n, n)
    conn = np.concatenate([np.column_stack([np.moveaxis(idx, a, 0)[:-1].ravel(), np.moveaxis(idx, a, 0)[1:].ravel()])
                           for a in range(3)]).astype(np.int64)
    ne = len(conn)
    sec = np.empty((ne, 10))
    sec[:, 0] = 0.01 * rng.uniform(0.5, 2, ne)
    sec[:, 2], sec[:, 3] = 1e-5 * rng.uniform(0.5, 2, ne), 2e-5 * rng.uniform(0.5, 2, ne)
    sec[:, 1] = sec[:, 2] + sec[:, 3]
    sec[:, 4] = 2.5e-5
    sec[:, 5:7] = 0.008 if case["timoshenko"] else np.inf
    sec[:, 7:] = rng.normal(size=(ne, 3))
    u1 = rng.uniform(-0.01, 0.01, (n ** 3, 3))
    a = rng.normal(scale=0.05, size=(n ** 3, 3))
    th = np.linalg.norm(a, axis=1)[:, None, None]
    S = np.zeros((n ** 3, 3, 3))
    S[:, 2, 1], S[:, 0, 2], S[:, 1, 0] = a[:, 0], a[:, 1], a[:, 2]
    S = S - S.transpose(0, 2, 1)
    R = np.eye(3) + np.sin(th) / th * S + (1 - np.cos(th)) / th ** 2 * (S @ S)
    return np.asfortranarray(xyz), np.ascontiguousarray(conn), sec, np.asfortranarray(u1), R


def _explicit_inputs(case, seed):
    """The plate (simply supported), the initial velocity, the load and the step."""
    n = case["n"]
    xyz, conn = _plate(case["el"], n, n, seed, False, jitter=0.05)
    fixed = np.zeros((len(xyz), 6), bool)
    fixed[_edge(xyz), 2] = True
    dof, nfree = _number(fixed)
    rng = np.random.Generator(np.random.PCG64(seed + 1))
    x, y = xyz[:, 0], xyz[:, 1]
    w = dof[:, 2]
    free = w <= nfree
    shape = np.sin(np.pi * x[free]) * np.sin(np.pi * y[free])
    V0 = np.zeros(nfree)
    V0[w[free] - 1] = 1e-3 * shape + rng.normal(0, 1e-5, free.sum())
    Fmag = np.zeros(nfree)
    Fmag[w[free] - 1] = 1e3 * shape / n ** 2
    dt = 0.3 / n / math.sqrt(E / RHO / (1 - NU ** 2))  # under the critical step 2 / omega_max
    g = np.sin(2 * np.pi * 50.0 * dt * np.arange(case["steps"] + 1)) if case["load"] else None
    return xyz, conn, dof, nfree, V0, Fmag, g, dt


# ---------------------------------------------------------------------------
# the program's side
# ---------------------------------------------------------------------------
def _fields(xyz, dof, nfree):
    geom0 = F.NodalField(xyz)
    dchi = F.NodalField(np.zeros((len(xyz), 6)))
    dchi.dofnums = dof
    dchi.nfreedofs = nfree
    return geom0, dchi


def _femm_class(el):
    return F.FEMMShellT3FF if el == "t3" else F.FEMMShellQ4RS


def _steel():
    return F.materials.MatDeforElastIso(E, NU, RHO)


def _call_inputs(case, seed):
    """The clamped wavy plate of the small analyses."""
    xyz, conn = _plate(case["el"], case["nx"], case["ny"], seed, True)
    fixed = np.zeros((len(xyz), 6), bool)
    fixed[xyz[:, 0] < 1e-9, :] = True
    dof, nfree = _number(fixed)
    return xyz, conn, dof, nfree, 0.01


def prepare(case, seed):
    s = dict(case)
    kind = case["kind"]
    if kind in ("call", "model"):
        xyz, conn, dof, nfree, t = _call_inputs(case, seed)
        s["geom0"], s["dchi"] = _fields(xyz, dof, nfree)
        s["femm"] = _femm_class(case["el"])(conn, t, _steel())
        s["nfree"] = nfree
        if kind == "call":
            s["femm"].associategeometry(s["geom0"])
        return s
    if kind == "explicit":
        xyz, conn, dof, nfree, V0, Fmag, g, dt = _explicit_inputs(case, seed)
        geom0, dchi = _fields(xyz, dof, nfree)
        femm = _femm_class(case["el"])(conn, 0.01, _steel())
        femm.associategeometry(geom0)
        M = femm.mass(F.SysmatAssemblerFFBlock(F.SysmatAssemblerSparseDiag(), nfree), geom0, dchi).diagonal()
        nnz = ctypes.c_int64()
        femm.ctx.call("fs_stiffness", _abi.FS_FP64, _abi.FS_ASM_SPARSE, nfree, ctypes.byref(nnz))
        C = (2 * 0.01 * 2 * np.pi * 50.0) * M
        s.update(femm=femm, cd=F.CentralDifference(femm, M, C, dt, PRECISION[case["precision"]]),
                 V0=V0, zero=np.zeros(nfree), Fmag=Fmag, g=g)
        return s
    ctx = Context(0)
    s["ctx"] = ctx
    if kind == "beams":
        xyz, conn, sec, u1, R = _beams(case, seed)
        nn, ne = len(xyz), len(conn)
        dof = np.asfortranarray(np.arange(1, 6 * nn + 1, dtype=np.int64).reshape(nn, 6))
        secs = (_abi.fs_beam_section * ne)()
        ctypes.memmove(secs, sec.ctypes.data, sec.nbytes)
        R1 = np.asfortranarray(R.transpose(0, 2, 1).reshape(nn, 9))
        ctx.call("fs_mesh_set", _abi.FS_COROTBEAM, nn, ptr(xyz), ne, ptr(conn), None, ptr(dof))
        ctx.call("fs_beam_setup", secs, 2.1e11, 0.3, RHO)
        ctx.call("fs_beam_state_set", ptr(u1), ptr(R1), None)
        s["n"] = 6 * nn
        s["nnz"] = ctypes.c_int64()
        return s
    if kind == "panels":
        Dps, Dt = F.materials.shell_material_stiffness(F.materials.MatDeforElastIso(4.32e8, 0.0))
        ctx.call("fs_params_set", _abi.make_params(Dps, Dt, 0.0, 0.0), None)
        panels = _panels(case, seed)
        k, vp, i64 = len(panels), ctypes.c_void_p, ctypes.c_int64
        dofs = [np.asfortranarray(np.arange(1, p[0].size * 2 + 1, dtype=np.int64).reshape(-1, 6)) for p in panels]
        arr = lambda vals, t: (t * k)(*vals)  # noqa: E731
        ctx.call("fs_batch_set", _abi.FS_T3FF, k, arr([len(p[0]) for p in panels], i64),
                 arr([p[0].ctypes.data for p in panels], vp), arr([len(p[1]) for p in panels], i64),
                 arr([p[1].ctypes.data for p in panels], vp), arr([d.ctypes.data for d in dofs], vp),
                 arr([d.size for d in dofs], i64), arr([p[2] for p in panels], ctypes.c_double))
        return s
    xyz, conn, dof, t = _assembly_inputs(case, seed)
    et = {("t3", False): _abi.FS_T3FF, ("t3", True): _abi.FS_T3FFCOMP, ("q4", False): _abi.FS_Q4RS,
          ("q4", True): _abi.FS_Q4RSCOMP}[(case["el"], case["layered"])]
    order = group = None
    if case["layered"]:
        group = _groups(len(conn))
        order = np.ascontiguousarray(np.argsort(group, kind="stable") + 1)
    ctx.call("fs_mesh_set", et, len(xyz), ptr(xyz), len(conn), ptr(conn), ptr(order), ptr(dof))
    Dps, Dt = F.materials.shell_material_stiffness(_steel())
    ctx.call("fs_params_set", _abi.make_params(Dps, Dt, RHO, t, quads=case["el"] == "q4"), None)
    if case["layered"]:
        Dps, Dts, rho, tp, layups = _layup()
        gs = [F.laminate([dict(Dps=Dps, Dts=Dts, thickness=tp, angle=a, rho=rho) for a in lay]) for lay in layups]
        ctx.call("fs_layups_set", len(gs), (_abi.fs_layup_group * len(gs))(*gs), ptr(group))
    ctx.call("fs_normals_compute")
    s["n"] = dof.size
    s["nnz"] = ctypes.c_int64()
    ctx.call("fs_pattern", s["n"], ctypes.byref(s["nnz"]))
    return s


def _assembly_inputs(case, seed):
    xyz, conn = _plate(case["el"], case["nx"], case["ny"], seed, case["wave"])
    dof = np.asfortranarray(np.arange(1, 6 * len(xyz) + 1, dtype=np.int64).reshape(-1, 6))
    return xyz, conn, dof, 0.005


def _groups(ne):
    """Layup group of each element: strips of 100 elements in turn."""
    return np.ascontiguousarray((np.arange(ne) // 100 % 2).astype(np.int32))


class _View:
    """A device array of the library for torch (no copy); it belongs to the
    context, which lives as long as the array is in use."""

    def __init__(self, ctx, address, count, kind):
        self.ctx = ctx
        self.__cuda_array_interface__ = {"shape": (count,), "typestr": kind, "data": (address, False), "version": 3}


def _matrix(ctx, pattern):
    """The matrix just assembled, on the device: values, and columns and row pointers too."""
    rp, ci, v = ctypes.c_void_p(), ctypes.c_void_p(), ctypes.c_void_p()
    n, nnz = ctypes.c_int64(), ctypes.c_int64()
    ctx.call("fs_matrix_device", ctypes.byref(rp), ctypes.byref(ci), ctypes.byref(v), ctypes.byref(n),
             ctypes.byref(nnz))
    out = [torch.as_tensor(_View(ctx, v.value, nnz.value, "<f8"), device="cuda")]
    if pattern:
        out.append(torch.as_tensor(_View(ctx, ci.value, nnz.value, "<i4"), device="cuda"))
        out.append(torch.as_tensor(_View(ctx, rp.value, n.value + 1, "<i8"), device="cuda"))
    return out


def run(s):
    kind = s["kind"]
    if kind == "call":
        K = s["femm"].stiffness(s["geom0"], None, None, s["dchi"])
        return [K.data, K.indices, K.indptr]
    if kind == "model":
        femm, geom0, dchi = s["femm"], s["geom0"], s["dchi"]
        femm.associategeometry(geom0)
        M = femm.mass(F.SysmatAssemblerFFBlock(F.SysmatAssemblerSparseDiag(), s["nfree"]), geom0, dchi)
        K = femm.stiffness(F.SysmatAssemblerFFBlock(F.SysmatAssemblerSparse(), s["nfree"]), geom0, None, None, dchi)
        return [K.data, M.data, K.indices, K.indptr]
    if kind == "explicit":
        cd = s["cd"]
        cd.set_state(s["zero"], s["V0"], s["zero"])
        if s["g"] is not None:
            cd.set_load(s["Fmag"], s["g"], s["steps"])
        cd.run(s["steps"])
        return list(cd.state())
    ctx = s["ctx"]
    if kind == "panels":
        ctx.call("fs_batch_stiffness", PRECISION[s["precision"]], _abi.FS_ASM_SPARSE, None)
        return _matrix(ctx, False)
    if kind == "beams":
        ctx.call("fs_beam_matrix", _abi.FS_BEAM_STIFFNESS, 1, _abi.FS_ASM_SPARSE, s["n"], ctypes.byref(s["nnz"]))
        return _matrix(ctx, False)
    ctx.call("fs_stiffness", PRECISION[s["precision"]], ASSEMBLER[s["assembler"]], s["n"], ctypes.byref(s["nnz"]))
    return _matrix(ctx, s["assembler"] == "symm")


# ---------------------------------------------------------------------------
# the work of a pass
# ---------------------------------------------------------------------------
def _counts(el, nx, ny):
    """elements, nodes, stored node blocks of a plate"""
    edges = nx * (ny + 1) + ny * (nx + 1) + nx * ny * (1 if el == "t3" else 2)
    nodes = (nx + 1) * (ny + 1)
    return nx * ny * (2 if el == "t3" else 1), nodes, nodes + 2 * edges


def _shell_work(el, ne, nodes, blocks, layered=False):
    """Inputs of the elements and nodes once, the values once; the Gram products
    of the upper node blocks, two operations each."""
    nen = 3 if el == "t3" else 4
    rows = 8 if el == "t3" else 32
    gram = rows * (nen * (nen + 1) // 2 * 36)
    if not layered:
        gram -= 3 * (rows // 8) * (nen * (nen + 1) // 2) * 27
    return {"bytes": ne * (4 * nen + 8) + nodes * 49 + blocks * 36 * 8, "flops": 2 * gram * ne}


def work(case):
    kind = case["kind"]
    if kind in ("call", "model", "assembly"):
        return _shell_work(case["el"], *_counts(case["el"], case["nx"], case["ny"]), case.get("layered", False))
    if kind == "panels":
        sizes = np.random.Generator(np.random.PCG64(3))
        tot = np.zeros(3, dtype=np.int64)
        for _ in range(case["panels"]):
            n = int(sizes.integers(16, case["nmax"] + 1))
            tot += _counts("t3", n, n)
        return _shell_work("t3", *[int(v) for v in tot])
    if kind == "explicit":
        # every step: the stored values of K, the state read and written once
        _, nodes, blocks = _counts(case["el"], case["n"], case["n"])
        size = {"fp64": 8, "mixed": 4, "comp": 6}[case["precision"]]
        return {"bytes": case["steps"] * (blocks * (36 * size + 4) + 6 * nodes * 8 * 12),
                "flops": case["steps"] * blocks * 72}
    n = case["n"]
    ne, nodes = 3 * n * n * (n - 1), n ** 3
    return {"bytes": ne * (8 + 80) + nodes * (24 + 24 + 72) + (nodes + 2 * ne) * 288, "flops": ne * 3 * 36 * 6 * 2}


# ---------------------------------------------------------------------------
# the same in 64 bits, dense
# ---------------------------------------------------------------------------
_GP = 0.577350269189626  # abscissa of the 2 x 2 Gauss rule


def _frame(a, b):
    e0 = a / a.norm(dim=-1, keepdim=True)
    e2 = torch.linalg.cross(e0, b)
    e2 = e2 / e2.norm(dim=-1, keepdim=True)
    return torch.stack([e0, torch.linalg.cross(e2, e0), e2], -2)


def _rotation(a):
    """Rotation matrices of the vectors a (angle |a|)."""
    x = (a * a).sum(-1)
    phi = x.sqrt()
    safe = phi.clamp_min(1e-150)
    s = torch.where(phi > 0, torch.sin(phi) / safe, torch.ones_like(phi))
    h = torch.where(phi > 0, torch.sin(phi / 2) / (safe / 2), torch.ones_like(phi))
    S = torch.zeros(a.shape[:-1] + (3, 3), dtype=a.dtype, device=a.device)
    S[..., 2, 1], S[..., 0, 2], S[..., 1, 0] = a[..., 0], a[..., 1], a[..., 2]
    S = S - S.transpose(-1, -2)
    return torch.eye(3, dtype=a.dtype, device=a.device) + s[..., None, None] * S + (h * h / 2)[..., None, None] * (S @ S)


def _dbasis(xi, eta):
    return torch.tensor([[-(1 - eta), -(1 - xi)], [1 - eta, -(1 + xi)], [1 + eta, 1 + xi], [-(1 + eta), 1 - xi]],
                        dtype=torch.float64, device="cuda") / 4


def _normals(X3, conn, el, csn):
    """Nodal normals and validity: X3 (nodes, 3), conn 0-based; csn: the layup
    normal of every element (layered), or None."""
    X = X3[conn]
    nen = conn.shape[1]
    per = []
    for a in range(nen):
        if el == "t3":
            J0, J1 = X[:, 1] - X[:, 0], X[:, 2] - X[:, 0]
        else:
            g = _dbasis([-1.0, 1.0, 1.0, -1.0][a], [-1.0, -1.0, 1.0, 1.0][a])
            J0, J1 = torch.einsum("eac,a->ec", X, g[:, 0]), torch.einsum("eac,a->ec", X, g[:, 1])
        n = torch.linalg.cross(J0, J1)
        size = n.norm(dim=-1, keepdim=True)
        per.append(((csn if csn is not None else n / size) * (size if el == "q4" else 1.0)))
    nrm = torch.zeros_like(X3)
    for a in range(nen):
        nrm.index_add_(0, conn[:, a], per[a])
    nrm = nrm / nrm.norm(dim=-1, keepdim=True)
    s = math.sin(30 / 180 * math.pi)
    cos_thr = 1 - (1 - math.sqrt(1 - s * s))
    bad = torch.zeros(len(X3), dtype=torch.int32, device=X3.device)
    for a in range(nen):
        if el == "t3":
            J0, J1 = X[:, 1] - X[:, 0], X[:, 2] - X[:, 0]
            n = torch.linalg.cross(J0, J1)  # the element's own normal, layered or not
        else:
            n = per[a]
        n = n / n.norm(dim=-1, keepdim=True)
        if el == "t3" and csn is not None:
            n = csn
        bad.index_add_(0, conn[:, a], ((nrm[conn[:, a]] * n).sum(-1) < cos_thr).to(torch.int32))
    return nrm, bad == 0


def _strain_map(e, nrm, valid, g):
    """Element-frame dofs (u, v, w, thx, thy of every node) from the global ones:
    Q (elements, 5 nen, 6 nen); also t (nodal triads in global components) and
    the rotation blocks."""
    ne, nen = nrm.shape[:2]
    a = torch.zeros_like(nrm)
    a[..., 0] = -torch.einsum("ec,eic->ei", e[:, 1], nrm) * valid
    a[..., 1] = torch.einsum("ec,eic->ei", e[:, 0], nrm) * valid
    A = _rotation(a)
    t = torch.einsum("eirk,erc->eikc", A, e)
    inv33 = 1 / A[..., 2, 2]
    m = A[..., :2, 2] * inv33[..., None]
    R2 = A[..., :2, :2] - inv33[..., None, None] * A[..., :2, 2, None] * A[..., None, :2, 2]
    W = 0.5 * (torch.einsum("ej,eik,ejkc->eijc", g[..., 0], A[..., 1, :], t)
               - torch.einsum("ej,eik,ejkc->eijc", g[..., 1], A[..., 0, :], t))
    Q = torch.zeros(ne, nen, 5, nen, 6, dtype=torch.float64, device=e.device)
    for i in range(nen):
        Q[:, i, :3, i, :3] = e
        Q[:, i, 3:, i, 3:] = torch.einsum("erl,elc->erc", R2[:, i], t[:, i, :2])
        Q[:, i, 3:, :, :3] = m[:, i, :, None, None] * W[:, i, None]
    return Q.reshape(ne, 5 * nen, 6 * nen), t, R2


def _bending_rows(g):
    ne, nen = g.shape[:2]
    B = torch.zeros(ne, 6, nen, 5, dtype=torch.float64, device=g.device)
    gx, gy = g[..., 0], g[..., 1]
    B[:, 0, :, 0] = gx
    B[:, 1, :, 1] = gy
    B[:, 2, :, 0], B[:, 2, :, 1] = gy, gx
    B[:, 3, :, 4] = gx
    B[:, 4, :, 3] = -gy
    B[:, 5, :, 3], B[:, 5, :, 4] = -gx, gy
    return B.reshape(ne, 6, 5 * nen)


def _layup_rotate(e, cs, B, Bs):
    M = torch.einsum("erc,eck->erk", e[:, :2], cs[:, :, :2])
    M = M / M.norm(dim=1, keepdim=True)
    m = (M[:, 0, 0] + M[:, 1, 1]) / 2
    d = (M[:, 0, 1] - M[:, 1, 0]) / 2
    n = torch.where(d >= 0, 1.0, -1.0).double() * (1 - m * m).clamp_min(0).sqrt()
    T = torch.stack([m * m, n * n, -m * n, n * n, m * m, m * n, 2 * m * n, -2 * m * n, m * m - n * n], -1).view(-1, 3, 3)
    Ts = torch.stack([m, -n, n, m], -1).view(-1, 2, 2)
    return torch.cat([T @ B[:, :3], T @ B[:, 3:]], 1), Ts @ Bs


def _t3_matrices(X, nrm, valid, c):
    J0, J1 = X[:, 1] - X[:, 0], X[:, 2] - X[:, 0]
    e = _frame(J0, J1)
    a, b = (J0 * e[:, 0]).sum(-1), (J0 * e[:, 1]).sum(-1)
    cc, d = (J1 * e[:, 0]).sum(-1), (J1 * e[:, 1]).sum(-1)
    Jd = a * d - b * cc
    Ae = Jd / 2
    g = torch.stack([torch.stack([b - d, d, -b], -1), torch.stack([cc - a, -cc, a], -1)], -1) / Jd[:, None, None]
    x, y = torch.stack([0 * a, a, cc], -1), torch.stack([0 * b, b, d], -1)
    Bs = torch.zeros(len(X), 2, 3, 5, dtype=torch.float64, device=X.device)
    for s, p, q in ((0, 1, 2), (1, 2, 0), (2, 0, 1)):  # the node orderings averaged
        pa, pb, pc, pd = x[:, p] - x[:, s], y[:, p] - y[:, s], x[:, q] - x[:, s], y[:, q] - y[:, s]
        k = 1 / (6 * Ae)
        Bs[:, 0, s, 2] += k * (pb - pd)
        Bs[:, 1, s, 2] += k * (pc - pa)
        Bs[:, 0, s, 4] += k * Ae
        Bs[:, 1, s, 3] -= k * Ae
        Bs[:, 0, p, 2] += k * pd
        Bs[:, 1, p, 2] -= k * pc
        Bs[:, 0, p, 3] -= k * pb * pd / 2
        Bs[:, 1, p, 3] += k * pb * pc / 2
        Bs[:, 0, p, 4] += k * pa * pd / 2
        Bs[:, 1, p, 4] -= k * pa * pc / 2
        Bs[:, 0, q, 2] -= k * pb
        Bs[:, 1, q, 2] += k * pa
        Bs[:, 0, q, 3] += k * pb * pd / 2
        Bs[:, 1, q, 3] -= k * pa * pd / 2
        Bs[:, 0, q, 4] -= k * pb * pc / 2
        Bs[:, 1, q, 4] += k * pa * pc / 2
    Bs = Bs.reshape(len(X), 2, 15)
    B = _bending_rows(g)
    t = c["t"]
    stab = t * t / (t * t + STAB["t3"] * 2 * Ae)
    if "cs" in c:
        B, Bs = _layup_rotate(e, c["cs"], B, Bs)
    D6, D2 = _moduli(c, len(X))
    Ke = Ae[:, None, None] * (B.transpose(1, 2) @ D6 @ B) + (Ae * stab)[:, None, None] * (Bs.transpose(1, 2) @ D2 @ Bs)
    Q, tn, R2 = _strain_map(e, nrm, valid, g)
    K = Q.transpose(1, 2) @ Ke @ Q
    Kt = torch.stack([Ke[:, 5 * i + 3:5 * i + 5, 5 * i + 3:5 * i + 5] for i in range(3)], 1)
    kavg = torch.einsum("eirl,eirs,eisl->e", R2, Kt, R2) / 6
    for i in range(3):
        n2 = tn[:, i, 2]
        K[:, 6 * i + 3:6 * i + 6, 6 * i + 3:6 * i + 6] += (kavg * valid[:, i])[:, None, None] * n2[:, :, None] * n2[:, None, :]
    return K


def _moduli(c, ne):
    """[tA tB; tB tD] with its integrals through the thickness, and the shear moduli."""
    if "cs" in c:
        return c["ABD"], c["H"]
    t = torch.as_tensor(c["t"], dtype=torch.float64, device="cuda").expand(ne)
    D6 = torch.zeros(ne, 6, 6, dtype=torch.float64, device="cuda")
    D6[:, :3, :3] = t[:, None, None] * c["Dps"]
    D6[:, 3:, 3:] = (t ** 3 / 12)[:, None, None] * c["Dps"]
    return D6, t[:, None, None] * (5 / 6) * c["Dt"]


def _q4_matrices(X, nrm, valid, c):
    ne = len(X)
    Xr = X - X.mean(1, keepdim=True)
    t = c["t"]
    stab = t * t / (t * t + STAB["q4"] * ((X - X[:, :1]) ** 2).sum(-1).amax(-1))
    D6, D2 = _moduli(c, ne)
    K = torch.zeros(ne, 24, 24, dtype=torch.float64, device=X.device)
    for xi, eta in ((-_GP, -_GP), (-_GP, _GP), (_GP, -_GP), (_GP, _GP)):
        dN = _dbasis(xi, eta)
        J = torch.einsum("eac,ak->eck", Xr, dN)
        e = _frame(J[..., 0], J[..., 1])
        Jac = torch.linalg.cross(J[..., 0], J[..., 1]).norm(dim=-1)
        J2 = torch.einsum("erc,eck->erk", e[:, :2], J)
        g = torch.einsum("ak,ekr->ear", dN, torch.linalg.inv(J2))
        P = torch.einsum("eac,erc->era", Xr, e[:, :2])
        x, y = P[:, 0], P[:, 1]
        r, s = xi, eta
        J11 = (x[:, 0] * (s - 1) - x[:, 1] * (s - 1) + x[:, 2] * (s + 1) - x[:, 3] * (s + 1)) / 4
        J21 = (y[:, 0] * (s - 1) - y[:, 1] * (s - 1) + y[:, 2] * (s + 1) - y[:, 3] * (s + 1)) / 4
        J12 = (x[:, 0] * (r - 1) - x[:, 1] * (r + 1) + x[:, 2] * (r + 1) - x[:, 3] * (r - 1)) / 4
        J22 = (y[:, 0] * (r - 1) - y[:, 1] * (r + 1) + y[:, 2] * (r + 1) - y[:, 3] * (r - 1)) / 4
        la, lb = torch.hypot(J11, J21), torch.hypot(J12, J22)
        det = J11 * J22 - J12 * J21
        Ax, Ay = x[:, 0] - x[:, 1] - x[:, 2] + x[:, 3], y[:, 0] - y[:, 1] - y[:, 2] + y[:, 3]
        Bx, By = x[:, 0] - x[:, 1] + x[:, 2] - x[:, 3], y[:, 0] - y[:, 1] + y[:, 2] - y[:, 3]
        Cx, Cy = x[:, 0] + x[:, 1] - x[:, 2] - x[:, 3], y[:, 0] + y[:, 1] - y[:, 2] - y[:, 3]
        LA, LB = torch.hypot(Ax + Bx * s, Ay + By * s), torch.hypot(Bx * r + Cx, By * r + Cy)
        one = torch.ones_like(det)
        x03, x12, x01, x23 = x[:, 0] - x[:, 3], x[:, 1] - x[:, 2], x[:, 0] - x[:, 1], x[:, 2] - x[:, 3]
        y03, y12, y01, y23 = y[:, 0] - y[:, 3], y[:, 1] - y[:, 2], y[:, 0] - y[:, 1], y[:, 2] - y[:, 3]
        rp, rm, sp, sm = r + 1, r - 1, s + 1, s - 1
        fa = torch.stack([torch.stack([rp * one, -rm * one, rm * one, -rp * one], -1) * 2,
                          torch.stack([-y03 * rp, y12 * rm, y12 * rm, -y03 * rp], -1),
                          torch.stack([x03 * rp, -x12 * rm, -x12 * rm, x03 * rp], -1)], -1)
        fb = torch.stack([torch.stack([-sp * one, sp * one, -sm * one, sm * one], -1) * 2,
                          torch.stack([y01 * sp, y01 * sp, y23 * sm, y23 * sm], -1),
                          torch.stack([-x01 * sp, -x01 * sp, -x23 * sm, -x23 * sm], -1)], -1)
        Bs = torch.zeros(ne, 2, 4, 5, dtype=torch.float64, device=X.device)
        for row, (pa, pb) in enumerate(((J21 / la, J22 / lb), (-J11 / la, -J12 / lb))):
            Bs[:, row, :, 2:] = ((pa * LA)[:, None, None] * fa + (pb * LB)[:, None, None] * fb) / (32 * det)[:, None, None]
        Bs = Bs.reshape(ne, 2, 20)
        B = _bending_rows(g)
        if "cs" in c:
            B, Bs = _layup_rotate(e, c["cs"], B, Bs)
        Ke = Jac[:, None, None] * (B.transpose(1, 2) @ D6 @ B) + (Jac * stab)[:, None, None] * (Bs.transpose(1, 2) @ D2 @ Bs)
        Q, _, _ = _strain_map(e, nrm, valid, g)
        K += Q.transpose(1, 2) @ Ke @ Q
    trace = []
    for i in range(4):
        Kr = K[:, 6 * i + 3:6 * i + 6, 6 * i + 3:6 * i + 6]
        trace.append((Kr.diagonal(dim1=1, dim2=2).sum(-1) - torch.einsum("ec,ecd,ed->e", nrm[:, i], Kr, nrm[:, i])) / 2)
    trace = torch.stack(trace, 1).clamp_min(0) * valid
    kavg = trace.sum(1) / valid.sum(1).clamp_min(1)
    for i in range(4):
        n = nrm[:, i]
        K[:, 6 * i + 3:6 * i + 6, 6 * i + 3:6 * i + 6] += (kavg * valid[:, i])[:, None, None] * n[:, :, None] * n[:, None, :]
    return K


def _beam_matrices(x0, xt, R, sec):
    def complete(f0, v):
        f2 = torch.linalg.cross(f0, v)
        f2 = f2 / f2.norm(dim=-1, keepdim=True)
        return torch.stack([f0, torch.linalg.cross(f2, f0), f2], -1)
    d0, d1 = x0[:, 1] - x0[:, 0], xt[:, 1] - xt[:, 0]
    L = d1.norm(dim=-1)
    F0 = complete(d0 / d0.norm(dim=-1, keepdim=True), sec[:, 7:])
    v = ((R[:, 0] + R[:, 1]) @ F0)[:, :, 1]
    Ft = complete(d1 / L[:, None], v)
    Em, G = 2.1e11, 2.1e11 / 2 / 1.3
    A, I2, I3, Jt, A2, A3 = (sec[:, k] for k in (0, 2, 3, 4, 5, 6))
    DN = torch.stack([Em * A / L, Em * I3 / L, 3 * Em * I3 / L / (1 + 12 * Em * I3 / (G * A2 * L * L)), Em * I2 / L,
                      3 * Em * I2 / L / (1 + 12 * Em * I2 / (G * A3 * L * L)), G * Jt / L], -1)
    a = torch.zeros(len(L), 6, 4, 3, dtype=torch.float64, device=L.device)
    a[:, 0, 0, 0], a[:, 0, 2, 0] = -1, 1
    a[:, 1, 1, 2], a[:, 1, 3, 2] = 1, -1
    a[:, 2, 0, 1], a[:, 2, 1, 2], a[:, 2, 2, 1], a[:, 2, 3, 2] = 2 / L, 1, -2 / L, 1
    a[:, 3, 1, 1], a[:, 3, 3, 1] = -1, 1
    a[:, 4, 0, 2], a[:, 4, 1, 1], a[:, 4, 2, 2], a[:, 4, 3, 1] = 2 / L, -1, -2 / L, -1
    a[:, 5, 1, 0], a[:, 5, 3, 0] = -1, 1
    g = torch.einsum("ecj,ekpj->ekpc", Ft, a).reshape(-1, 6, 12)
    return torch.einsum("eki,ek,ekj->eij", g, DN, g)


def _assembled(conn, nnodes, dof, n, matrices, chunk=1 << 17):
    """CSR values (rows and columns 1..n in order) of the element matrices that
    matrices(i, j) gives for elements i..j, and the columns and row pointers."""
    ne, nen = conn.shape
    pair = (conn[:, :, None] * nnodes + conn[:, None, :]).reshape(-1)
    key, slot = torch.unique(pair, return_inverse=True)
    slot = slot.view(ne, nen * nen)
    blk = torch.zeros(len(key), 6, 6, dtype=torch.float64, device=conn.device)
    for i in range(0, ne, chunk):
        j = min(ne, i + chunk)
        K = matrices(i, j).reshape(j - i, nen, 6, nen, 6).transpose(2, 3).reshape(-1, 6, 6)
        blk.index_add_(0, slot[i:j].reshape(-1), K)
    row = dof[key // nnodes][:, :, None].expand(-1, 6, 6).reshape(-1)
    col = dof[key % nnodes][:, None, :].expand(-1, 6, 6).reshape(-1)
    val = blk.reshape(-1)
    keep = (row <= n) & (col <= n)
    if not bool(keep.all()):
        row, col, val = row[keep], col[keep], val[keep]
    order = torch.argsort((row - 1) * n + (col - 1))
    rowptr = torch.zeros(n + 1, dtype=torch.int64, device=conn.device)
    rowptr[1:] = torch.cumsum(torch.bincount(row - 1, minlength=n), 0)
    return val[order], col[order] - 1, rowptr


def _shell_exact(el, xyz, conn, dof, n, t, Dps, Dt, layered=False):
    """t: a thickness, or one per element (panels)."""
    dev = lambda v: torch.as_tensor(np.ascontiguousarray(v)).cuda()  # noqa: E731
    X3, cn, dof = dev(xyz), dev(conn) - 1, dev(dof)
    c = {"Dps": dev(Dps), "Dt": dev(Dt)}
    csn = group = None
    if layered:
        Pps, Pts, _, tp, layups = _layup()
        red = [_laminate(Pps, Pts, tp, lay) for lay in layups]
        group = dev(_groups(len(conn))).long()
        ABD, H = dev(np.stack([r[0] for r in red])), dev(np.stack([r[1] for r in red]))
        thick = dev(np.array([tp * len(lay) for lay in layups]))
        csn = torch.tensor([0.0, 0.0, 1.0], dtype=torch.float64, device="cuda").expand(len(conn), 3)
    nrm, valid = _normals(X3, cn, el, csn)
    tv = None if np.isscalar(t) else dev(t)
    f = _t3_matrices if el == "t3" else _q4_matrices

    def matrices(i, j):
        p = cn[i:j]
        k = dict(c, t=t if tv is None else tv[i:j])
        if layered:
            gr = group[i:j]
            k.update(ABD=ABD[gr], H=H[gr], t=thick[gr],
                     cs=torch.eye(3, dtype=torch.float64, device="cuda").expand(j - i, 3, 3))
        return f(X3[p], nrm[p], valid[p].double(), k)
    return _assembled(cn, len(xyz), dof, n, matrices, 1 << (17 if el == "t3" else 16))


def _laminate(Dps, Dts, tp, angles):
    """[A B; B D] and H of a layup (parabolic shear factor)."""
    A, B, D, H = np.zeros((3, 3)), np.zeros((3, 3)), np.zeros((3, 3)), np.zeros((2, 2))
    T = tp * len(angles)
    z = -T / 2
    for deg in angles:
        a = math.radians(deg)
        m, n = math.cos(a), -math.sin(a)
        R = np.array([[m * m, n * n, 2 * m * n], [n * n, m * m, -2 * m * n], [-m * n, m * n, m * m - n * n]])
        Q = R @ Dps @ R.T
        c, s = math.cos(a), math.sin(a)
        S = np.array([[c, -s], [s, c]])
        Hp = S.T @ Dts @ S
        z1 = z + tp
        A += (z1 - z) * Q
        B += (z1 ** 2 - z ** 2) / 2 * Q
        D += (z1 ** 3 - z ** 3) / 3 * Q
        H += 5 / 4 * (z1 - z - 4 / 3 * (z1 ** 3 - z ** 3) / T ** 2) * Hp
        z = z1
    return np.block([[A, B], [B, D]]), H


def _plane(young, nu):
    q = young / (1 - nu * nu)
    Dps = np.array([[q, nu * q, 0], [nu * q, q, 0], [0, 0, young / 2 / (1 + nu)]])
    return Dps, np.eye(2) * (young / 2 / (1 + nu))


def _lumped(el, xyz, conn, t, dof, n):
    """The lumped mass diagonal."""
    X = xyz[conn - 1]
    if el == "t3":
        area = np.linalg.norm(np.cross(X[:, 1] - X[:, 0], X[:, 2] - X[:, 0]), axis=1) / 2
    else:
        area = 0.0
        for xi, eta in ((-_GP, -_GP), (-_GP, _GP), (_GP, -_GP), (_GP, _GP)):
            dN = _dbasis(xi, eta).cpu().numpy()
            J = np.einsum("eac,ak->eck", X, dN)
            area = area + np.linalg.norm(np.cross(J[..., 0], J[..., 1]), axis=1)
    share = np.zeros(len(xyz))
    for a in range(conn.shape[1]):
        np.add.at(share, conn[:, a] - 1, RHO * t * area / conn.shape[1])
    m = np.empty(dof.size)
    m[dof[:, :3].ravel() - 1] = np.repeat(share, 3)
    m[dof[:, 3:].ravel() - 1] = np.repeat(share * t * t / 12, 3)
    return m[:n]


def exact(case, seed):
    kind = case["kind"]
    Dps, Dt = _plane(E, NU)
    if kind in ("call", "model"):
        xyz, conn, dof, nfree, t = _call_inputs(case, seed)
        n = nfree if kind == "model" else dof.size
        val, _, _ = _shell_exact(case["el"], xyz, conn, dof, n, t, Dps, Dt)
        if kind == "call":
            return [val[val != 0], None, None]
        return [val, _lumped(case["el"], xyz, conn, t, dof, n), None, None]
    if kind == "assembly":
        xyz, conn, dof, t = _assembly_inputs(case, seed)
        val, _, _ = _shell_exact(case["el"], xyz, conn, dof, dof.size, t, Dps, Dt, case["layered"])
        return [val[val != 0], None, None] if case["assembler"] == "symm" else [val]
    if kind == "panels":
        xs, cs, ts, off = [], [], [], 0
        for xyz, conn, t in _panels(case, seed):
            xs.append(xyz)
            cs.append(conn + off)
            ts.append(np.full(len(conn), t))
            off += len(xyz)
        xyz = np.concatenate(xs)
        dof = np.arange(1, 6 * len(xyz) + 1, dtype=np.int64).reshape(-1, 6)
        Dps, Dt = _plane(4.32e8, 0.0)
        return [_shell_exact("t3", xyz, np.concatenate(cs), dof, dof.size, np.concatenate(ts), Dps, Dt)[0]]
    if kind == "beams":
        xyz, conn, sec, u1, R = _beams(case, seed)
        dev = lambda v: torch.as_tensor(np.ascontiguousarray(v)).cuda()  # noqa: E731
        X, U, Rt, cn, sc = dev(xyz), dev(u1), dev(R), dev(conn) - 1, dev(sec)
        dof = torch.arange(1, 6 * len(xyz) + 1, device="cuda").view(-1, 6)
        return [_assembled(cn, len(xyz), dof, dof.numel(), lambda i, j: _beam_matrices(
            X[cn[i:j]], (X + U)[cn[i:j]], Rt[cn[i:j]], sc[i:j]))[0]]
    xyz, conn, dof, nfree, V0, Fmag, g, dt = _explicit_inputs(case, seed)
    val, col, rowptr = _shell_exact(case["el"], xyz, conn, dof, nfree, 0.01, Dps, Dt)
    K = torch.sparse_csr_tensor(rowptr, col, val, size=(nfree, nfree))
    dev = lambda v: torch.as_tensor(v).cuda()  # noqa: E731
    M = dev(_lumped(case["el"], xyz, conn, 0.01, dof, nfree))
    C = (2 * 0.01 * 2 * np.pi * 50.0) * M
    invMC = 1 / (M + dt / 2 * C)
    U, V, A = torch.zeros_like(M), dev(V0), torch.zeros_like(M)
    load = dev(Fmag)
    for k in range(case["steps"]):
        U = U + dt * V + dt * dt / 2 * A
        f = -(K @ U) - C * (V + dt / 2 * A)
        if g is not None:
            f = f + g[k + 1] * load
        V = V + dt / 2 * A
        A = invMC * f
        V = V + dt / 2 * A
    return [U, V, A]
