"""Extremes of the rotated y' from the atoms outside a polygon of the
structure: structures at the sizes where one block's preparation hands over to
the many-block one, and point sets without an interior (one atom, a line,
coincident atoms, a ring), against the oracle.  Voxel indices are compared
bit-exact, intensities by normwise relative L2 error <= 1e-5."""
import numpy as np
import pytest

from giwaxsim_gb300 import forward as F
from oracle import giwaxs_oracle as O

pytestmark = pytest.mark.gpu
RTOL = 1e-5
R, DQ, MAX_Q = 0.5, 0.15, 1.5
PHIS = np.array([0.0, 17.0, 45.0, 90.0, 133.5, 179.0])


def points(shape, n):
    rng = np.random.default_rng(n)
    if shape == "cloud":
        return rng.uniform(0.0, 1.0, (n, 3)) * [14.0, 11.0, 9.0] + [-300.0, 50.0, 7.0]
    if shape == "line":
        return np.linspace(0.0, 1.0, n)[:, None] * [9.0, -7.0, 4.0]
    if shape == "one place":
        return np.tile([[3.0, -2.0, 1.0]], (n, 1))
    if shape == "grid":  # ties on every face
        return np.argwhere(np.ones((n, n, n))) * 0.5
    if shape == "tall":  # higher and wider than the grid: atoms outside it
        return rng.uniform(0.0, 1.0, (n, 3)) * [30.0, 45.0, 60.0]
    a = np.linspace(0.0, 2 * np.pi, n, endpoint=False)  # ring
    return np.stack([6.0 * np.cos(a), 6.0 * np.sin(a), a], axis=1)


@pytest.mark.parametrize("shape,n", [
    ("cloud", 1), ("cloud", 2), ("cloud", 3), ("cloud", 33), ("cloud", 2047),
    ("cloud", 2048), ("cloud", 2049), ("cloud", 9001), ("line", 7), ("line", 2051),
    ("one place", 5), ("one place", 2500), ("grid", 12), ("grid", 14), ("ring", 700),
    ("ring", 4099), ("tall", 600), ("tall", 3001)])
def test_extremes_vs_oracle(shape, n):
    xyz = points(shape, n)
    fv = np.full(len(xyz), 6.0 + 0j)
    geom = F.VoxelGeometry(R, DQ, MAX_Q)
    other = points("cloud", 2300)[:len(xyz)] + 1.0
    structures = [(xyz, fv, None), (other, np.full(len(other), 5.0 + 0j), None)]
    fill = bool(np.ptp(xyz, axis=0).all())  # (no box to average over otherwise)
    plan = F.VoxelPlan(geom, structures, phis=PHIS, fill_bkg=fill, smooth=0)
    try:
        plan.set_atoms()
        for _ in range(2):  # the second pass starts from the first one's state
            plan.execute()
        for k, phi in enumerate(PHIS):
            y, z = plan.debug_deposit(k)
            _, info = O.project_slice(xyz, fv, phi, geom.grid_size, R, 0j, 1, 1, 1, False, 0)
            ok = info["valid"]
            want_y, want_z = np.full(len(xyz), -1), np.full(len(xyz), -1)
            want_y[ok], want_z[ok] = info["y_idx"], info["z_idx"]
            assert np.array_equal(y, want_y) and np.array_equal(z, want_z), phi
        ref = O.voxelgrid([s[:2] for s in structures], R, DQ, MAX_Q, PHIS, fill, 0)
        assert np.linalg.norm(plan.iq() - ref["iq"]) <= RTOL * np.linalg.norm(ref["iq"])
    finally:
        plan.close()
