"""Beam elements beyond the range of the quotients by reciprocals on the GPU
(infinite section properties, no length) among ordinary ones: every
element matrix and vector has the host build's finite entries, infinities and
NaN, and the ordinary elements keep their bits.  Tolerance 1e-12 of the largest
finite entry."""
import numpy as np
import pytest

import beams as BM
from flexshell import _abi, beam as B
from flexshell.femm import NodalField
from hostcheck import hostmath as HC

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("which", [_abi.FS_BEAM_STIFFNESS, _abi.FS_BEAM_GEOSTIFFNESS, _abi.FS_BEAM_MASS])
def test_odd_elements_among_ordinary_ones(which):
    xyz, conn, sec, u1, R1, v1, dof, nf = BM.lattice_frame()
    mat = BM.Material(2.1e3, 0.3, 7.8)
    good = B.FEMMCorotBeam(conn, sec, mat)
    want = good.element_matrices(which, NodalField(xyz), u1, R1, v1)
    good.close()
    odd = sec.copy()
    odd[3, 0] = np.inf
    odd[7, 4] = np.inf
    odd[8, 2] = np.inf
    odd[20, 3] = np.inf
    odd[40, 0] = 1e300
    conn2 = conn.copy()
    conn2[30, 1] = conn2[30, 0]   # no length
    femm = B.FEMMCorotBeam(conn2, odd, mat)
    G = femm.element_matrices(which, NodalField(xyz), u1, R1, v1)
    femm.close()
    rest = np.setdiff1d(np.arange(len(conn)), [3, 7, 8, 20, 30, 40])
    assert np.array_equal(G[rest], want[rest])
    H = HC.beam_elements(which, xyz, conn2, odd, mat.E, mat.nu, mat.rho, u1, R1, v1)
    for e in (3, 7, 8, 20, 30, 40):
        g, h = G[e], H[e]
        fin = np.isfinite(h)
        assert np.array_equal(np.isfinite(g), fin)
        if fin.any():
            assert np.abs(g[fin] - h[fin]).max() <= 1e-12 * np.abs(h[fin]).max()
    if which == _abi.FS_BEAM_STIFFNESS:
        assert not np.isfinite(G[[3, 7, 8, 20, 30]]).any()
