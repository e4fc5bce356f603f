"""When VoxelPlan asks for the real-grid path: the phase of a caller's average
voxel f (constants) must be that of the f values, as the path takes the grids'
phase from it."""
import numpy as np
import pytest

from giwaxsim_gb300 import forward as F

GEOM = (0.5, 0.15, 1.5)


def params(constants=None, real=None, f=6.0 + 0.2j):
    xyz = np.random.default_rng(1).uniform(0.0, 12.0, (50, 3))
    items = [(xyz, np.full(50, f), None), (xyz + 1.0, np.full(50, -2.0 * f), None)]
    return F.VoxelPlan(F.VoxelGeometry(*GEOM), items, phis=np.array([0.0, 30.0]),
                       constants=constants, real=real, ctx=object(), create=False).params


def const(avg1, avg2):
    return [(12.0, 11.0, 10.0, avg1), (12.0, 11.0, 10.0, avg2)]


@pytest.mark.parametrize("real", [None, True])
@pytest.mark.parametrize("a,b,want", [
    (0.6 + 0.02j, 1.2 + 0.04j, 1), (-0.3 - 0.01j, 0.6 + 0.02j, 1),
    (0.6 + 0j, 1.2 + 0.04j, 0), (0.6 + 0.02j, 1.2 - 0.04j, 0), (0.6 + 0.02j, 0.04 + 1.2j, 0)])
def test_phase_of_the_constants(real, a, b, want):
    assert params(const(a, b), real).real_grids == want


def test_without_constants():
    assert params().real_grids == 1
    assert params(real=False).real_grids == 0
    assert params(const(0.6 + 0.02j, 1.2 + 0.04j), real=False).real_grids == 0
