"""The y extremes at the block shapes the other tests do not reach: four
slices a block (more slices than four a multiprocessor) with blocks that hold
the slices of two or three structures and a partial last one, and a slice's
candidates shared by several blocks (hollow structures: most atoms are
candidates), with structures on both sides of the line in one plan.  Deposit
indices bit-exact against the oracle."""
import numpy as np
import pytest

from giwaxsim_gb300 import forward as F
from oracle import giwaxs_oracle as O

pytestmark = pytest.mark.gpu
R, DQ, MAX_Q = 0.5, 0.15, 1.5


def structure(shape, n):
    rng = np.random.default_rng(n)
    if shape == "box":
        return rng.uniform(0.0, 1.0, (n, 3)) * [14.0, 11.0, 9.0] + [40.0, -50.0, 7.0]
    if shape == "tall":  # higher and wider than the grid: atoms outside it
        return rng.uniform(0.0, 1.0, (n, 3)) * [30.0, 45.0, 60.0]
    a = rng.uniform(0.0, 2 * np.pi, n)  # tube: every atom on the hull; pipe: wider
    R0 = 6.0 if shape == "tube" else 25.0  # than the grid
    return np.stack([R0 * np.cos(a), R0 * np.sin(a), rng.uniform(0.0, 9.0, n)], axis=1)


def multiprocessors():
    torch = pytest.importorskip("torch")
    return torch.cuda.get_device_properties(0).multi_processor_count


@pytest.mark.parametrize("shapes", [
    [("box", 700), ("box", 33), ("box", 1), ("box", 2047)],      # one-block preparation
    [("box", 700), ("tube", 2500), ("box", 9001), ("box", 5)],   # many-block preparation
    [("tube", 4096), ("box", 6000), ("tube", 4097), ("tube", 12301), ("box", 40)],
    [("box", 50), ("tube", 17001), ("tall", 16385)],
    [("pipe", 17003), ("box", 5000), ("pipe", 300)],
    [("tube", 4097)]])
@pytest.mark.parametrize("per_sm", [0, 2, 4])
def test_blocks_of_slices_vs_oracle(shapes, per_sm):
    # angles not divisible by four, a total that is not either
    n_phi = per_sm * multiprocessors() // len(shapes) + 7
    while n_phi % 4 == 0 or n_phi * len(shapes) % 4 == 0:
        n_phi += 1
        if len(shapes) % 4 == 0 and n_phi % 4:
            break
    n = n_phi * len(shapes)
    assert n > per_sm * multiprocessors()
    phis = np.linspace(0.0, 179.0, n_phi)
    items = []
    for shape, count in shapes:
        xyz = structure(shape, count)
        items.append((xyz, np.full(len(xyz), 6.0 + 0j), None))
    geom = F.VoxelGeometry(R, DQ, MAX_Q)
    plan = F.VoxelPlan(geom, items, phis=phis, real=False)
    try:
        plan.set_atoms()
        for _ in range(2):
            plan.execute()
        look = {0, 1, 2, 3, n // 2, n - 1, n - 2, n - 3, n - 4}
        for t in range(1, len(items)):  # both sides of a structure's first slice
            look |= set(range(t * n_phi - 4, t * n_phi + 4))
        for sl in sorted(look):
            xyz, fv, _ = items[sl // n_phi]
            y, z = plan.debug_deposit(sl)
            _, info = O.project_slice(xyz, fv, phis[sl % n_phi], geom.grid_size, R, 0j, 1, 1, 1,
                                      False, 0)
            ok = info["valid"]
            want_y, want_z = np.full(len(xyz), -1), np.full(len(xyz), -1)
            want_y[ok], want_z[ok] = info["y_idx"], info["z_idx"]
            assert np.array_equal(y, want_y) and np.array_equal(z, want_z), sl
    finally:
        plan.close()
