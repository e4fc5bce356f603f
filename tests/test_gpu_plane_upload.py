"""Plane mode takes only the plane of I(q) it reads: images with the fixed
axis x, y or z, from host and device arrays, uneven shapes and a full replay
list, against the general path on the whole array."""
import ctypes

import numpy as np
import pytest

from giwaxsim_gb300 import _native as N

pytestmark = pytest.mark.gpu

# base plane x = 0; y and z take its place
INIT = {"x": np.eye(3), "y": np.array([[0, 1, 0], [1, 0, 0], [0, 0, 1]], float),
        "z": np.array([[0, 0, 1], [0, 1, 0], [1, 0, 0]], float)}


def turns(axis, n):
    """n rotations about a coordinate axis, that axis' row and column exact."""
    i, j = [k for k in range(3) if k != "xyz".index(axis)]
    out = []
    for a in np.linspace(0.1, 3.0, n):
        R = np.eye(3)
        R[i, i] = R[j, j] = np.cos(a)
        R[i, j], R[j, i] = -np.sin(a), np.sin(a)
        out.append(R)
    return np.array(out)


def image(iq, axis, n_or, pixels, no_plane, on_device=False):
    import torch
    ctx = N.default_context()
    p = N.DetectorParams()
    p.n_h, p.n_v = pixels
    for k in range(3):
        p.iq_shape[k] = iq.shape[k]
    p.qmin_x, p.qmin_y, p.qmin_z, p.dq = -1.0, -0.9, -1.1, 0.05
    p.mirror, p.accum, p.exact, p.no_plane = 0, N.GW_ACCUM_FP64, 0, int(no_plane)
    h, v = np.linspace(-1, 1, pixels[0]), np.linspace(-0.8, 1.1, pixels[1])
    init = np.ascontiguousarray(INIT[axis].reshape(1, 9))
    rot = np.ascontiguousarray(turns(axis, n_or).reshape(-1, 9))
    nrot = np.ones(n_or, np.int32)
    w = np.linspace(0.1, 1.0, n_or)
    plan = ctypes.c_void_p()
    lib = N.lib()
    N.check(lib.gw_detector_plan_create(ctx.handle, ctypes.byref(p), N.ptr(h), N.ptr(v),
                                        N.ptr(init), 1, N.ptr(nrot), N.ptr(rot), N.ptr(w),
                                        n_or, ctypes.byref(plan)))
    try:
        if on_device:
            d = torch.as_tensor(iq).cuda()
            torch.cuda.synchronize()
            N.check(lib.gw_detector_set_iq(plan, ctypes.c_void_p(d.data_ptr()), 1))
        else:
            N.check(lib.gw_detector_set_iq(plan, N.ptr(iq), 0))
        out = np.empty((pixels[1], pixels[0]))
        for _ in range(2):
            N.check(lib.gw_detector_execute(plan))
            N.check(lib.gw_detector_get(plan, N.ptr(out), 0))
        return out
    finally:
        lib.gw_detector_plan_destroy(plan)


@pytest.mark.parametrize("axis", ["x", "y", "z"])
@pytest.mark.parametrize("shape", [(37, 41, 45), (1, 5, 3), (300, 260, 7)])
@pytest.mark.parametrize("cap", [None, "1"])
def test_plane_vs_whole(axis, shape, cap, monkeypatch):
    if cap:
        monkeypatch.setenv("GW_DET_WORKLIST_CAP", cap)
    iq = np.random.default_rng(5).exponential(1e4, shape)
    pixels = (65, 33)
    ref = image(iq, axis, 9, pixels, True)
    # both sum the same float32 samples; replayed ones are added in float64
    # in scheduling order
    for on_device in (False, True):
        got = image(iq, axis, 9, pixels, False, on_device)
        assert np.allclose(got, ref, rtol=1e-6, atol=0)
