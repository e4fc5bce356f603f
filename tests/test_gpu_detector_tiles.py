"""Detector images of the fast kernels against the all-exact kernel at the
edges of pixel tiles, of the batches and groups of orientations and of the
chunks they are staged in, with room in the worklist and without.

Samples and weights are positive, so every pixel's float32 partial sums (at
most 16 fused adds each, then float64) and the weight's rounding to float32
are off by at most 17 * 2^-24 of the pixel; one more for the products of
these errors."""
import numpy as np
import pytest

from giwaxsim_gb300 import forward as F

pytestmark = pytest.mark.gpu
TOL = 18 * 2.0 ** -24


def images(npx, n, plane, exact):
    rng = np.random.default_rng(17 * npx + n)
    q = np.linspace(-1.6, 1.6, 41)
    iq = rng.uniform(0.1, 1.0, (41, 41, 41))
    one = np.ones(1)
    angles, w = np.linspace(0.0, 170.0, n), rng.uniform(0.5, 1.5, n)
    turn = (angles, w, np.zeros(1), one) if plane else (np.array([11.0]), one, angles, w)
    plan = F.DetectorPlan(iq.shape, q, q, q, npx, 1.5, (90.0, 0, 0), ("psi", "None", "None"),
                          *turn, np.zeros(1), one, False, exact=exact)
    plan.set_iq(iq)
    plan.execute()
    image = plan.result()
    plan.close()
    return image


@pytest.mark.parametrize("cap", [None, "3"])
@pytest.mark.parametrize("plane", [True, False])
@pytest.mark.parametrize("npx", [2, 15, 16, 17, 33])
@pytest.mark.parametrize("n", [1, 7, 8, 9, 17, 137])
def test_tile_and_batch_edges(npx, n, plane, cap, monkeypatch):
    if cap:
        monkeypatch.setenv("GW_DET_WORKLIST_CAP", cap)
    got, ref = images(npx, n, plane, False), images(npx, n, plane, True)
    assert ref.min() > 0
    assert np.all(np.abs(got - ref) <= TOL * ref)
