"""The detector gather at the limits of its index arithmetic: an axis fixed at
an index beyond the float32 floors' range, a plane of lines more than 2^31 bytes
apart, and a volume of more than 2^32 elements, against the exact path
(float64 indices of every sample)."""
import numpy as np
import pytest

from giwaxsim_gb300 import forward as F

pytestmark = pytest.mark.gpu


def plans(shape, q, psis, phis=(0.0,), **kw):
    """The fast and the exact plan; q: (x, y, z) axes of an I(q) of shape
    (ny, nx, nz)."""
    one = lambda a: np.full(len(a), 1.0 / len(a))  # noqa: E731
    for exact in (False, True):
        yield F.DetectorPlan(shape, *q, 64, 1.0, (), (), psis, one(psis), phis, one(phis), [0.0],
                             [1.0], mirror=False, exact=exact, **kw)


@pytest.mark.parametrize("kw", [dict(plane=False), dict(accum="kahan32"), dict()])
def test_fixed_axis_beyond_the_exact_floors(kw):
    """x = 0 lies at index 4,500,001 of the x axis; the adjoint too."""
    n, dq = 4500010, 1e-4
    qx = (np.arange(n) - 4500001.5) * dq
    shape = (2, n, 2)
    iq = np.random.default_rng(1).random(shape)
    psis = np.linspace(0.0, 90.0, 7)
    g = np.random.default_rng(2).standard_normal((64, 64))
    img, adj = [], []
    # (dq is the z axis': 2 voxels a side along y and z)
    qz = np.array([-dq, 0.0])
    for plan in plans(shape, (qx, qz, qz), psis, **kw):
        try:
            plan.set_iq(iq)
            plan.execute()
            img.append(plan.result())
            adj.append(plan.backward(g))
        finally:
            plan.close()
    assert np.allclose(img[0], img[1], rtol=1e-6, atol=0)
    assert np.array_equal(adj[0] != 0, adj[1] != 0)
    assert np.allclose(adj[0], adj[1], rtol=1e-9, atol=1e-15)


def test_plane_of_lines_far_apart():
    """nx nz float64 values between the lines of the plane: more bytes than
    cudaDeviceProp::memPitch, which the plane's 2-D copy takes all the same."""
    ny, nx, nz = 3, 16385, 16390
    assert nx * nz * 8 > 2 ** 31
    iq = np.zeros((ny, nx, nz))  # (only the plane's pages are ever touched)
    fixed = 7
    iq[:, fixed, :] = np.random.default_rng(3).random((ny, nz))
    dq = 1e-4
    qx = (np.arange(nx) - fixed - 0.5) * dq
    qy = np.array([-1.5, -0.5, 0.5]) * dq
    qz = (np.arange(nz) - nz / 2) * dq
    psis = np.linspace(0.0, 90.0, 5)
    w = np.full(5, 0.2)
    plan = F.DetectorPlan(iq.shape, qx, qy, qz, 64, 1.0, (), (), psis, w, [0.0], [1.0], [0.0],
                          [1.0], mirror=False)
    try:
        plan.set_iq(iq)
        plan.execute()
        img = plan.result()
        idx = [plan.debug_indices(o) for o in range(5)]
    finally:
        plan.close()
    want = sum(0.2 * iq.reshape(-1)[i] for i in idx).reshape(64, 64)
    want = np.where(want <= 0, 1e-6, want) * 1e-6
    assert np.allclose(img, want, rtol=1e-6, atol=0)


@pytest.mark.parametrize("accum", ["fp64", "kahan32"])
@pytest.mark.parametrize("phis", [(0.0,), (0.0, 25.0, 71.0)])
def test_volume_of_more_than_32_bit_indices(accum, phis):
    """2^32 elements and more, the samples at the volume's end; the gather and
    the exact path on the same device array."""
    torch = pytest.importorskip("torch")
    n = 1626
    assert n ** 3 > 2 ** 32
    if torch.cuda.mem_get_info()[0] < 40 << 30:
        pytest.skip("needs a 17 GB array")
    iq = torch.empty((n, n, n), dtype=torch.float32, device="cuda")
    line = torch.arange(n * n, device="cuda", dtype=torch.int64).reshape(n, n)
    for y in range(n):
        iq[y] = ((line + 977 * y) % 1009).float()
    torch.cuda.synchronize()
    dq = 0.002
    q = (np.arange(n) - 0.8 * n) * dq  # q = 0 (and the pixels) towards the end
    img = []
    for plan in plans((n, n, n), (q, q, q), np.linspace(0.0, 80.0, 5), phis, accum=accum,
                      plane=False):
        try:
            plan.set_iq_device32(iq.data_ptr())
            plan.execute()
            img.append(plan.result())
        finally:
            plan.close()
    del iq
    torch.cuda.empty_cache()
    assert np.allclose(img[0], img[1], rtol=1e-5, atol=0)
