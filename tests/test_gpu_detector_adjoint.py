"""The detector's adjoint at the edges of its pixel tiles and of its splits of
the orientations, against a float64 scatter at the forward's indices.

Both sides sum the same products in float64 in another order: a voxel of T
terms is off by at most 2 T 2^-53 of the sum of their magnitudes."""
import numpy as np
import pytest

from giwaxsim_gb300 import forward as F

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("plane", [True, False])
@pytest.mark.parametrize("npx", [2, 15, 16, 17, 32, 33, 65])
@pytest.mark.parametrize("n", [1, 8, 9, 67])
def test_adjoint_scatter(npx, n, plane):
    rng = np.random.default_rng(17 * npx + n)
    q = np.linspace(-1.6, 1.6, 31)
    iq = rng.uniform(0.1, 1.0, (31, 31, 31))
    one, zero = np.ones(1), np.zeros(1)
    angles, w = np.linspace(0.0, 170.0, n), rng.uniform(0.5, 1.5, n)
    turn = (angles, w, zero, one) if plane else (np.array([11.0]), one, angles, w)
    plan = F.DetectorPlan(iq.shape, q, q, q, npx, 1.5, (90.0, 0, 0), ("psi", "None", "None"),
                          *turn, zero, one, False)
    plan.set_iq(iq)
    plan.execute()
    g = rng.standard_normal((npx, npx)) * (rng.random((npx, npx)) > 0.2)
    got = plan.backward(g)
    ref, mag, terms = (np.zeros(iq.size) for _ in range(3))
    for o in range(n):
        idx = plan.debug_indices(o).ravel()
        np.add.at(ref, idx, 1e-6 * g.ravel() * w[o])
        np.add.at(mag, idx, np.abs(1e-6 * g.ravel() * w[o]))
        np.add.at(terms, idx, 1.0)
    plan.close()
    assert np.all(np.abs(got.ravel() - ref) <= 2 * (terms + 2) * 2.0 ** -53 * mag)
