"""Real-grid plans whose window is wider than half the transform buffer (two
window rows of floats share one buffer of complex values) against the general
path, at transform lengths from 128 to 2048, and what such plans still take
that narrower real-grid plans refuse: per-shell f values and the adjoint."""
import numpy as np
import pytest

from giwaxsim_gb300 import _native as N
from giwaxsim_gb300 import forward as F

pytestmark = pytest.mark.gpu
RTOL = 1e-5

# (r, dq, max_q, box edge), transform length
CASES = [((0.4, 0.1, 0.6), 22.0, 128), ((0.3, 0.08, 0.4), 45.0, 256),
         ((0.2, 0.05, 0.3), 70.0, 640), ((0.15, 0.04, 0.3), 80.0, 1024),
         ((0.12, 0.04, 0.3), 90.0, 1280), ((0.1, 0.04, 0.3), 100.0, 1536),
         ((0.1, 0.035, 0.25), 130.0, 2048)]
PHIS = np.array([0.0, 11.0, 45.0, 90.0, 133.5])


def ldm(m):
    return m + m // 16 + 4


def atoms(box, seed, n=301):
    rng = np.random.default_rng(seed)
    xyz = rng.uniform(0.0, box, (n, 3)) * [1.0, 0.97, 0.3]
    return xyz, np.where(rng.random(n) < 0.3, -0.5, 1.0) * (6.0 + 0.2j)


def rel_l2(a, b):
    return np.linalg.norm(a - b) / np.linalg.norm(b)


@pytest.mark.parametrize("axes,box,m", CASES)
@pytest.mark.parametrize("fill,smooth", [(False, 0), (True, 1.5)])
def test_wide_window_vs_general(axes, box, m, fill, smooth):
    geom = F.VoxelGeometry(*axes)
    xyz, fv = atoms(box, m)
    out = {}
    for real in (None, False):
        plan = F.VoxelPlan(geom, [(xyz, fv, None)], phis=PHIS, fill_bkg=fill,
                           smooth=smooth, real=real)
        try:
            info = plan.info()
            assert info["real"] == (real is None)
            assert 2 * info["Ly"] > ldm(info["My"]) and info["My"] == m
            plan.set_atoms()
            plan.execute()
            out[real] = plan.iq().copy()
        finally:
            plan.close()
    assert rel_l2(out[None], out[False]) <= RTOL


@pytest.mark.parametrize("binning", ["atomic", "gather"])
@pytest.mark.parametrize("what", ["adjoint", "shells"])
def test_wide_plan_takes_the_adjoint_and_shells(binning, what):
    axes, box, m = CASES[1]
    geom = F.VoxelGeometry(*axes)
    xyz, fv = atoms(box, 3)
    bound = 1.1 * np.sqrt(3) * geom.q[-1]
    g_iq = np.random.default_rng(4).standard_normal((geom.crop_hi - geom.crop_lo + 1,) * 3)
    got = {}
    for real in (None, False):
        plan = F.VoxelPlan(geom, [(xyz, fv, None)], phis=PHIS, real=real, binning=binning)
        try:
            plan.set_atoms()
            plan.execute()
            assert plan.info()["real"] == (real is None)
            if what == "adjoint":
                got[real] = [plan.backward(g_iq)["g_f"].view(float)]
                got[real].append(plan.iq().copy())  # of the execute before it
            else:
                avg = plan.structs["avg_f_re"][0] + 1j * plan.structs["avg_f_im"][0]
                plan.set_shells(geom.q, np.array([0.0]), np.array([bound]), 1.5 * fv[None, :],
                                np.full((1, 1), 1.5 * avg))
                plan.execute()
                got[real] = [plan.iq().copy()]
                plan.set_shells(None, None, None, None, None)
                plan.set_atoms()
            assert plan.info()["real"] == 0
            plan.execute()
            got[real].append(plan.iq().copy())
        finally:
            plan.close()
    for a, b in zip(got[None], got[False]):
        assert rel_l2(a, b) <= RTOL


@pytest.mark.parametrize("binning", ["atomic", "gather"])
def test_failed_change_of_path_leaves_the_plan(binning):
    """Every allocation on the way to the general path fails once: the plan
    still runs the real path (and its graph) with the same result."""
    axes, box, m = CASES[1]
    geom = F.VoxelGeometry(*axes)
    xyz, fv = atoms(box, 3)
    g_iq = np.random.default_rng(4).standard_normal((geom.crop_hi - geom.crop_lo + 1,) * 3)
    plan = F.VoxelPlan(geom, [(xyz, fv, None)], phis=PHIS, binning=binning)
    try:
        plan.set_atoms()
        plan.capture_graph()
        plan.execute()
        before, ref = plan.info(), plan.iq().copy()
        assert before["real"] == 1
        failed = 0
        while True:
            N.set_alloc_fault(failed)
            try:
                plan.backward(g_iq)
            except N.GwError as e:
                assert e.status == N.GW_ERR_OOM
            finally:
                N.set_alloc_fault(-1)
            if not plan.info()["real"]:
                break
            assert plan.info() == before
            failed += 1
            plan.execute()
            assert rel_l2(plan.iq(), ref) <= RTOL
        assert failed == (3 if binning == "atomic" else 12)
        after = plan.info()
        if binning == "atomic":  # F1 in and out, the row table out, the profiles in
            a, b = before, after
            nf = a["Nc"] + a["k0"]  # columns ky >= 0
            assert b["device_bytes"] - a["device_bytes"] == 8 * (
                b["batch"] * b["Lz"] * b["Nc"] - a["batch"] * a["Lz"] * nf
                - a["n_slices"] * a["Ly"]) + 12 * a["n_slices"] * a["Ly"]
        plan.execute()
        assert rel_l2(plan.iq(), ref) <= RTOL
    finally:
        plan.close()


def test_refused_calls_leave_the_plan():
    """A backward or set_shells that is refused, and a clear of the shells,
    keep a wide plan on the real path; a refusal keeps its graph too."""
    axes, box, m = CASES[1]
    geom = F.VoxelGeometry(*axes)
    xyz, fv = atoms(box, 3)
    g_iq = np.ones((geom.crop_hi - geom.crop_lo + 1,) * 3)
    for kw in (dict(average="separate"), dict(fill_bkg=True)):
        plan = F.VoxelPlan(geom, [(xyz, fv, None), (xyz + 1.0, fv, None)], phis=PHIS, **kw)
        try:
            plan.set_atoms()
            plan.capture_graph()
            before = plan.info()
            assert before["real"] == 1 and before["graph_kernels"] > 0
            with pytest.raises(N.GwError) as e:
                plan.backward(g_iq)
            assert e.value.status == N.GW_ERR_ARG
            with pytest.raises(N.GwError) as e:
                plan.backward(g_iq, want_xyz=True)
            assert e.value.status == N.GW_ERR_ARG
            for lower, upper in (([1.0], [0.5]), ([0.0, 0.1], [0.5, 0.4])):
                with pytest.raises(N.GwError) as e:
                    plan.set_shells(geom.q, np.array(lower), np.array(upper),
                                    np.ones((len(lower), 2 * len(xyz))), np.ones((len(lower), 2)))
                assert e.value.status == N.GW_ERR_ARG
            assert plan.info() == before
            plan.execute()
            plan.set_shells(None, None, None, None, None)
            assert plan.info()["real"] == 1
        finally:
            plan.close()
    # no atoms yet
    plan = F.VoxelPlan(geom, [(xyz, fv, None)], phis=PHIS)
    try:
        with pytest.raises(N.GwError) as e:
            plan.backward(g_iq)
        assert e.value.status == N.GW_ERR_STATE and plan.info()["real"] == 1
    finally:
        plan.close()


def test_gather_store_too_large_for_the_general_path(monkeypatch):
    """Gather binning asked for, with a pixel store that fits the limit with
    the columns ky >= 0 and not with all of them: a call that needs the
    general path is refused, again when it is repeated, and changes nothing."""
    axes, box, m = CASES[1]
    geom = F.VoxelGeometry(*axes)
    xyz, fv = atoms(box, 3)
    g_iq = np.ones((geom.crop_hi - geom.crop_lo + 1,) * 3)
    probe = F.VoxelPlan(geom, [(xyz, fv, None)], phis=PHIS, binning="atomic")
    i = probe.info()
    probe.close()
    per = (i["Nc"] + i["k0"]) * i["Nr"] * 4  # bytes a slice, columns ky >= 0
    phis = np.linspace(0.0, 179.0, int(0.9 * 2 ** 20 / per))
    assert len(phis) * i["Nc"] * i["Nr"] * 4 > 2 ** 20
    monkeypatch.setenv("GW_GATHER_MAX_MB", "1")
    plan = F.VoxelPlan(geom, [(xyz, fv, None)], phis=phis, binning="gather")
    try:
        plan.set_atoms()
        plan.execute()
        before, ref = plan.info(), plan.iq().copy()
        assert before["real"] == 1 and before["gather"] == 1
        for _ in range(2):
            with pytest.raises(N.GwError) as e:
                plan.backward(g_iq)
            assert e.value.status == N.GW_ERR_ARG
            assert "gw_voxel_backward" in str(e.value) and "GW_GATHER_MAX_MB" in str(e.value)
            assert plan.info() == before
            plan.execute()
            assert rel_l2(plan.iq(), ref) <= RTOL
    finally:
        plan.close()


@pytest.mark.parametrize("binning", ["atomic", "gather"])
def test_sums_of_the_last_execute_after_the_change_of_path(binning):
    """sums() and iq() asked for after a backward are those of the execute
    before it, not of the general path's empty pixel store."""
    axes, box, m = CASES[1]
    geom = F.VoxelGeometry(*axes)
    xyz, fv = atoms(box, 3)
    g_iq = np.ones((geom.crop_hi - geom.crop_lo + 1,) * 3)
    plan = F.VoxelPlan(geom, [(xyz, fv, None)], phis=PHIS, binning=binning)
    try:
        plan.set_atoms()
        plan.execute()
        ref = plan.sums(), plan.iq().copy()
        plan.execute()  # (nothing made on request yet)
        plan.backward(g_iq)
        assert plan.info()["real"] == 0
        for _ in range(2):
            assert rel_l2(plan.sums(), ref[0]) <= RTOL and rel_l2(plan.iq(), ref[1]) <= RTOL
            plan.execute()
    finally:
        plan.close()


def test_window_of_the_last_execute_after_the_change_of_path():
    """debug_window shows the last execute's deposit, before and after
    set_shells takes the plan to the general path."""
    axes, box, m = CASES[1]
    geom = F.VoxelGeometry(*axes)
    xyz, fv = atoms(box, 3)
    fv = fv * (3.0 - 4.0j)
    plan = F.VoxelPlan(geom, [(xyz, fv, None)], phis=PHIS)
    try:
        plan.set_atoms()
        plan.execute()
        assert plan.info()["real"] == 1
        ref = plan.debug_window(1)[0].copy()
        assert abs(ref.sum() - fv.sum()) <= RTOL * np.abs(fv).sum()
        plan.set_shells(geom.q, np.array([0.0]), np.array([2.0]), fv[None, :], np.ones((1, 1)))
        assert plan.info()["real"] == 0
        assert rel_l2(plan.debug_window(1)[0], ref) <= RTOL
        plan.execute()
        assert rel_l2(plan.debug_window(1)[0], ref) <= RTOL
    finally:
        plan.close()


def test_graph_captured_follows_the_change_of_path():
    axes, box, m = CASES[1]
    geom = F.VoxelGeometry(*axes)
    xyz, fv = atoms(box, 3)
    g_iq = np.ones((geom.crop_hi - geom.crop_lo + 1,) * 3)
    plan = F.VoxelPlan(geom, [(xyz, fv, None)], phis=PHIS)
    try:
        plan.set_atoms()
        plan.capture_graph()
        with pytest.raises(N.GwError):
            plan.backward(g_iq, want_xyz=True)  # refused
        assert plan.graph_captured
        plan.backward(g_iq)
        assert not plan.graph_captured
        plan.capture_graph()
        plan.backward(g_iq)  # on the general path already
        assert plan.graph_captured and plan.info()["graph_kernels"] > 0
    finally:
        plan.close()


@pytest.mark.parametrize("which,capture", [(0, False), (1, False), (1, True)])
def test_other_f_values_on_the_device(which, capture):
    """Device f values that are not real multiples of the average voxel f
    take a wide plan to the general path; multiples keep it and its graph."""
    torch = pytest.importorskip("torch")
    axes, box, m = CASES[2]
    geom = F.VoxelGeometry(*axes)
    (xyz, fv), (xyz2, fv2) = atoms(box, 3), atoms(0.9 * box, 4, 2500)
    items = [(xyz, fv, None), (xyz2, fv2 * 1j, None)]
    other = [fv.copy(), fv2 * 1j]
    other[which][7::11] *= 1.0 - 0.01j
    other = np.concatenate(other).astype(np.complex64)
    got = []
    for real in (None, False):
        plan = F.VoxelPlan(geom, items, phis=PHIS, smooth=1.0, real=real)
        try:
            x = torch.as_tensor(plan.xyz).cuda()
            good = torch.as_tensor(plan.f).cuda() * 1.5
            bad = torch.as_tensor(other.view(np.float32)).cuda()
            torch.cuda.synchronize()
            plan.set_atoms(x.data_ptr(), good.data_ptr(), on_device=True)
            plan.capture_graph()
            plan.set_atoms(x.data_ptr(), good.data_ptr(), on_device=True)
            plan.execute()
            assert plan.info()["real"] == (real is None) and plan.graph_captured
            got.append([plan.iq().copy()])
            if real is None:
                # set and not executed: nothing happens
                plan.set_atoms(x.data_ptr(), bad.data_ptr(), on_device=True)
                plan.set_atoms(x.data_ptr(), good.data_ptr(), on_device=True)
                plan.execute()
                assert plan.info()["real"] == 1 and rel_l2(plan.iq(), got[-1][0]) <= RTOL
                plan.set_atoms(x.data_ptr(), bad.data_ptr(), on_device=True)
                N.set_alloc_fault(0)
                try:
                    with pytest.raises(N.GwError) as e:
                        plan.execute()
                    assert e.value.status == N.GW_ERR_OOM
                finally:
                    N.set_alloc_fault(-1)
                for call in (plan.execute, plan.iq, plan.capture_graph):
                    with pytest.raises(N.GwError) as e:
                        call()
                    assert e.value.status == N.GW_ERR_STATE and plan.info()["real"] == 1
            plan.set_atoms(x.data_ptr(), bad.data_ptr(), on_device=True)
            if capture:
                if real is None:
                    N.set_alloc_fault(0)
                    try:
                        with pytest.raises(N.GwError) as e:
                            plan.capture_graph()
                        assert e.value.status == N.GW_ERR_OOM
                        with pytest.raises(N.GwError) as e:
                            plan.execute()  # (looks again)
                        assert e.value.status == N.GW_ERR_OOM
                    finally:
                        N.set_alloc_fault(-1)
                    plan.set_atoms(x.data_ptr(), bad.data_ptr(), on_device=True)
                plan.capture_graph()
                assert plan.info()["real"] == 0
            plan.execute()
            assert plan.info()["real"] == 0
            assert plan.graph_captured == (real is False or capture)
            got[-1].append(plan.iq().copy())
            plan.set_atoms(x.data_ptr(), good.data_ptr(), on_device=True)
            plan.execute()
            got[-1].append(plan.iq().copy())
        finally:
            plan.close()
    for a, b in zip(*got):
        assert rel_l2(a, b) <= RTOL
    assert rel_l2(got[1][1], got[1][0]) > 100 * RTOL


# (r, dq, max_q), box edge; transform lengths from 64 to 384, wide and narrow
SHORT = [((0.5, 0.15, 0.5), 8.0), ((0.4, 0.1, 0.6), 22.0), ((0.5, 0.15, 1.5), 13.0),
         ((0.3, 0.08, 0.4), 45.0), ((0.3, 0.06, 1.0), 50.0)]


@pytest.mark.parametrize("axes,box", SHORT)
@pytest.mark.parametrize("accum", ["fp64", "kahan32"])
def test_row_blocks_of_both_sizes(axes, box, accum):
    """Real rows in the smaller blocks (launches that would not fill the GPU)
    and in the others, several structures of uneven height (row pairs across two
    slices, an odd number of rows), plain and from a graph, against the general
    path."""
    torch = pytest.importorskip("torch")
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    geom = F.VoxelGeometry(*axes)
    items = [(xyz * [1.0, 1.0, z], fv, None) for (xyz, fv), z in
             ((atoms(box, 5), 1.0), (atoms(0.8 * box, 6, 90), 2.7), (atoms(0.9 * box, 7, 411), 0.31))]
    probe = F.VoxelPlan(geom, items, phis=PHIS)
    rows = probe.info()["Lz"]
    assert probe.info()["real"] == 1
    probe.close()
    # at most 16 sequences of two rows a block: four blocks a multiprocessor
    enough = 4 * sms * 2 * 16 // rows + 1
    for n_phi in (3, enough):
        phis = np.linspace(0.0, 178.0, n_phi)
        out = []
        for real in (None, False):
            plan = F.VoxelPlan(geom, items, phis=phis, fill_bkg=True, smooth=1.0, real=real,
                               accum=accum)
            try:
                plan.set_atoms()
                plan.execute()
                out.append(plan.iq().copy())
                plan.capture_graph()
                plan.execute()
                assert rel_l2(plan.iq(), out[-1]) <= RTOL
            finally:
                plan.close()
        assert rel_l2(*out) <= RTOL


@pytest.mark.parametrize("axes,box,m", CASES)
def test_wide_windows_of_uneven_structures(axes, box, m):
    """Row pairs across two slices, Kahan sums and a captured graph at every
    length."""
    geom = F.VoxelGeometry(*axes)
    items = [(xyz * [1.0, 1.0, z], fv, None) for (xyz, fv), z in
             ((atoms(box, 5), 1.0), (atoms(0.8 * box, 6, 90), 2.7))]
    out = []
    for real in (None, False):
        plan = F.VoxelPlan(geom, items, phis=PHIS, smooth=1.5, real=real, accum="kahan32")
        try:
            plan.set_atoms()
            plan.capture_graph()
            plan.execute()
            assert plan.info()["real"] == (real is None)
            out.append(plan.iq().copy())
        finally:
            plan.close()
    assert rel_l2(*out) <= RTOL
