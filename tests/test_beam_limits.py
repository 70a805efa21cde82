"""The beam stiffness at a double's limits, on the host: infinite or undefined
section properties give what the full sum of the stiffness terms gives, and so do
lengths and stiffnesses beyond the range of the quotients by reciprocals.
Tolerance of finite matrices: 1e-12 of the largest entry, the FP64 parity bound."""
import numpy as np
import pytest

from hostcheck import hostmath as HC


def _rows(x, e2):
    """The six 12-vectors g_k of a straight beam along x (its own frame), length L."""
    L = np.linalg.norm(x[1] - x[0])
    f0 = (x[1] - x[0]) / L
    f2 = np.cross(f0, e2)
    f2 /= np.linalg.norm(f2)
    f1 = np.cross(f2, f0)
    o = np.zeros(3)
    return L, np.array([np.r_[-f0, o, f0, o], np.r_[o, f2, o, -f2], np.r_[2 / L * f1, f2, -2 / L * f1, f2],
                        np.r_[o, -f1, o, f1], np.r_[2 / L * f2, -f1, -2 / L * f2, -f1], np.r_[o, -f0, o, f0]])


@pytest.mark.parametrize("what", ["A", "I2", "I3", "J", "nan A", "nan J", "none"])
@pytest.mark.parametrize("axis", [(1.0, 0, 0), (0.6, 0.0, 0.8), (0.3, -0.5, 0.7)])
def test_infinite_and_undefined_sections(what, axis):
    x = np.array([[0.0, 0, 0], axis])
    e2 = np.array([0.1, 1.0, 0.2])
    s = dict(A=2.0, I1=0.5, I2=0.3, I3=0.4, J=0.2)
    if what != "none":
        s[what.split()[-1]] = np.nan if what.startswith("nan") else np.inf
    sec = np.array([[s["A"], s["I1"], s["I2"], s["I3"], s["J"], np.inf, np.inf, *e2]])
    K = HC.beam_elements(0, x, np.array([[1, 2]]), sec, 10.0, 0.25)[0]
    L, g = _rows(x, e2)
    E, G = 10.0, 4.0
    with np.errstate(all="ignore"):
        DN = np.array([E * s["A"], E * s["I3"], 3 * E * s["I3"], E * s["I2"], 3 * E * s["I2"], G * s["J"]]) / L
        want = sum(DN[k] * g[k][:, None] * g[k][None, :] for k in range(6))
    if what == "none":
        assert np.abs(K - want).max() <= 1e-13 * np.abs(want).max()
        return
    # a zero times an infinity is undefined, whichever entry it is in
    assert not np.isfinite(want).any() and not np.isfinite(K).any()


@pytest.mark.parametrize("size,E", [(1e-285, 10.0), (1e-120, 1.0), (1.0, 1e-300), (1e100, 1.0), (1e150, 1e130),
                                    (1.0, 1e290), (1.0, 0.0)])
def test_sizes_beyond_the_quotients(size, E):
    # stiffnesses and lengths with quotients near a double's limits
    x = size * np.array([[0.0, 0, 0], [0.3, -0.5, 0.7]])
    e2 = np.array([0.1, 1.0, 0.2])
    a = min(size, 1.0)
    sec = np.array([[2.0 * a, 0.5, 0.3 * a, 0.4 * a, 0.2 * a, np.inf, np.inf, *e2]])
    K = HC.beam_elements(0, x, np.array([[1, 2]]), sec, E, 0.25)[0]
    with np.errstate(all="ignore"):
        L, g = _rows(x, e2)
        G = E / 2 / 1.25
        DN = np.array([E * sec[0, 0], E * sec[0, 3], 3 * E * sec[0, 3], E * sec[0, 2], 3 * E * sec[0, 2], G * sec[0, 4]]) / L
        want = sum(DN[k] * g[k][:, None] * g[k][None, :] for k in range(6))
    fin = np.isfinite(want)
    assert np.array_equal(np.isfinite(K), fin)
    if fin.any():
        assert np.abs(K[fin] - want[fin]).max() <= 1e-12 * np.abs(want[fin]).max()


def test_no_length():
    sec = np.array([[2.0, 0.5, 0.3, 0.4, 0.2, np.inf, np.inf, 0.1, 1.0, 0.2]])
    K = HC.beam_elements(0, np.zeros((2, 3)), np.array([[1, 2]]), sec, 10.0, 0.25)[0]
    assert np.isnan(K).all()
