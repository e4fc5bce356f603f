"""The detector's orientation list made axis by axis (orientation_matrices)
against one matrix at a time: the same matrices bit for bit, the same
rotation counts and weights."""
import numpy as np
import pytest

from giwaxsim_gb300 import forward as F


def one_by_one(corners, psis, pw, phis, hw, thetas, tw):
    n_rot, mats, weights = [], [], []
    for ps, w1 in zip(psis, pw):
        for ph, w2 in zip(phis, hw):
            for th, w3 in zip(thetas, tw):
                c, k = corners, 0
                for kind, ang in (("psi", ps), ("phi", ph), ("theta", th)):
                    R = c.matrix(kind, ang)
                    c = c.rotate(R)
                    if not np.array_equal(R, np.eye(3)):
                        mats.append(R)
                        k += 1
                n_rot.append(k)
                weights.append(w1 * w2 * w3)
    return np.array(n_rot), np.array(mats).reshape(-1, 3, 3), np.array(weights, float)


LISTS = [([0.0], [0.0], [0.0]), (np.linspace(0, 180, 13), [0.0], [0.0]),
         (np.linspace(0, 15, 4), np.linspace(0, 179, 7), [0.0]),
         ([0.0, 31.7], [0.0, -12.5, 90.0], [0.0, 3.25, 45.0]),
         ([0.0, 20.0], [0.0], [7.5]), (np.arange(3), np.arange(2), np.arange(2))]


@pytest.mark.parametrize("psis,phis,thetas", LISTS)
@pytest.mark.parametrize("init", [(), ("psi", 90.0), ("phi", 33.0)])
@pytest.mark.parametrize("wtype", [np.float64, np.float32])
def test_same_bits(psis, phis, thetas, init, wtype):
    psis, phis, thetas = (np.asarray(a) for a in (psis, phis, thetas))
    h = np.linspace(-2.3, 2.3, 51)
    c = F.PlaneCorners(h, h)
    if init:
        c = c.rotate(c.matrix(*init))
    rng = np.random.default_rng(1)
    w = [rng.random(len(a)).astype(wtype) for a in (psis, phis, thetas)]
    args = (psis, w[0], phis, w[1], thetas, w[2])
    n, m, wt = F.orientation_matrices(c, *args)
    n0, m0, w0 = one_by_one(c, *args)
    assert np.array_equal(n, n0)
    assert np.array_equal(m, m0)
    assert np.array_equal(wt, w0)


def test_degenerate_plane_and_unequal_lists():
    """One pixel (no edge to take an axis from) gives the matrices of no
    finite direction, and lists are cut to their weights, as one by one."""
    h = np.array([0.5])
    c = F.PlaneCorners(h, h)
    args = ([0.0, 10.0], [0.5, 0.5], [0.0], [1.0], [0.0], [1.0])
    with np.errstate(all="ignore"):
        n, m, _ = F.orientation_matrices(c, *args)
        n0, m0, _ = one_by_one(c, *args)
    assert np.array_equal(n, n0) and np.array_equal(m, m0, equal_nan=True)
    h = np.linspace(-1, 1, 5)
    n, m, w = F.orientation_matrices(F.PlaneCorners(h, h), [1.0, 2.0, 3.0], [0.5, 0.5],
                                     [0.0], [1.0], [], [])
    assert len(n) == len(m) == len(w) == 0


def test_weights_of_any_iterable():
    """Weights as zip takes them: generators, longer and mixed lists."""
    h = np.linspace(-1, 1, 5)
    c = F.PlaneCorners(h, h)
    psis, phis, thetas = [0.0, 10.0, 20.0], [5.0, 6.0], [0.0, 1.0]
    pw = [0.25, np.float32(0.1), 0.65]
    hw, tw = (np.float32(0.3), 0.7, 0.9), [1, 2]
    ref = one_by_one(c, psis, pw, phis, hw, thetas, tw)
    got = F.orientation_matrices(c, psis, (w for w in pw), phis, hw, thetas, iter(tw))
    for a, b in zip(got, ref):
        assert np.array_equal(a, b)

    def forever():
        while True:
            yield 0.5

    ref = one_by_one(c, psis, [0.5] * 3, phis, [0.5] * 2, thetas, [0.5] * 2)
    got = F.orientation_matrices(c, psis, forever(), phis, forever(), thetas, [0.5] * 9)
    for a, b in zip(got, ref):
        assert np.array_equal(a, b)
