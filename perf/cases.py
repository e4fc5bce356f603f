"""Performance cases of the GIWAXS forward path and its gradient.

Each case is one pass of a program that uses the framework, through its
public entry points.  The kinds:

  voxel     a VoxelPlan kept by the program (its graph captured), new atoms
            each pass: atoms on the device -> float32 I(q) on the device,
            where a detector plan or another GPU program reads it;
  detector  detectormaker_fitting on an I(q) array in host memory (one that
            was saved, or came from another program) -> detector image;
  simulate  the drop-in pair of a config run, voxelgridmaker_fitting and
            then detectormaker_fitting, on host arrays, every input its own
            structure; the image as float32, as pictures are kept;
  fit       SlabFit.images: the detector images of K slab sizes (one pass
            of the grid search), as a float32 stack;
  gradient  one training step of occupancies, smoothing and (bilinear
            deposit) coordinates against a target image, with PyTorch
            float32 parameters: their gradients.

exact() restates every kind in plain 64-bit torch and numpy: dense grids, a
full FFT per slice, every index as numpy's float64 arithmetic gives it.
"""
import math

import numpy as np
import torch

# f' + i f'' near 10 keV
F1F2 = {"C": 0.0192 + 0.0097j, "S": 0.3189 + 0.5567j, "F": 0.0732 + 0.0534j,
        "Si": 0.2541 + 0.3302j}
Z = {"C": 6, "F": 9, "Si": 14, "S": 16}
# carbon's Cromer-Mann coefficients (International Tables Vol. C 6.1.1.4)
F0_C = (2.31, 20.8439, 1.02, 10.2075, 1.5886, 0.5687, 0.865, 51.6512, 0.2156)
GRAPHITE = (2.46, 2.46, 6.70, 90.0, 90.0, 120.0)
ENERGY = 10000.0

VOXEL = dict(kind="voxel", structures=1, fill=False, smooth=0.0, accum="fp64")
DETECTOR = dict(kind="detector", init_psi=0.0, phis=1, thetas=1, mirror=True)
SIMULATE = dict(kind="simulate", fill=False, smooth=0.0, init_psi=0.0)


def listed():
    return [
        # a molecule-sized cluster at low resolution: a call of few
        # microseconds of work, where launches and latency count
        dict(VOXEL, name="voxel-cluster-13A", material="graphite", x=14.0, y=12.0, z=13.0,
             r=0.5, dq=0.15, max_q=1.5, slices=24),
        # a small crystal at everyday resolution
        dict(VOXEL, name="voxel-graphite-50A", material="graphite", x=50.0, y=50.0, z=50.0,
             r=0.3, dq=0.03, max_q=3.0, slices=180),
        # a large crystal with filled background and smoothing, one element
        dict(VOXEL, name="voxel-si-100A", material="silicon", x=100.0, y=100.0, z=100.0,
             r=0.25, dq=0.02, max_q=4.0, slices=360, fill=True, smooth=2.0),
        # a polymer slab of the shipped example's shape: three elements, flat
        # box, the automatic slice count, no background
        dict(VOXEL, name="voxel-polymer-176A", material="lamellar", x=176.0, y=43.0, z=186.0,
             r=0.3, dq=0.02, max_q=2.0, slices=889),
        # the largest: a polymer lamella at fine resolution
        dict(VOXEL, name="voxel-lamellar-200A", material="lamellar", x=200.0, y=200.0, z=200.0,
             r=0.2, dq=0.015, max_q=2.5, slices=720, fill=True, smooth=2.0),
        # an ensemble of crystallites of uneven size, averaged
        dict(VOXEL, name="voxel-ensemble-16", material="graphite", x=75.0, y=75.0, z=75.0,
             r=0.3, dq=0.03, max_q=3.0, slices=180, structures=16, smooth=1.0),
        # rotation about the beam: every sample lies in one plane of I(q)
        dict(DETECTOR, name="detector-psi-1000px", r=0.25, dq=0.02, max_q=4.0, pixels=1000,
             psis=91, psi_end=90.0, init_psi=90.0),
        # the shipped example's texture: 16 psi x 180 phi orientations
        dict(DETECTOR, name="detector-texture-500px", r=0.3, dq=0.02, max_q=2.0, pixels=500,
             psis=16, psi_end=15.0, phis=180, phi_end=179.0),
        # a whole config run on a large crystal, host arrays in and out
        dict(SIMULATE, name="simulate-si-100A", material="silicon", x=100.0, y=100.0, z=100.0,
             r=0.25, dq=0.02, max_q=4.0, slices=360, fill=True, smooth=2.0, pixels=1000,
             psis=91, psi_end=90.0, init_psi=90.0),
        # a round of a slab-size search
        dict(kind="fit", name="fit-graphite-5", r=0.3, dq=0.04, max_q=2.5, candidates=5, size=45.0,
             slices=120, smooth=1.0, pixels=301, psis=46, psi_end=90.0),
        # refinement of every occupancy and position of a crystal
        dict(kind="gradient", name="gradient-si-60A", material="silicon", x=60.0, y=60.0, z=60.0,
             r=0.3, dq=0.04095, max_q=3.0, slices=180, deposit="bilinear", sigma=1.2, pixels=512,
             psis=91, psi_end=90.0, checkpoint=16),
        # refinement of the occupancies of a polymer, nearest-bin deposit
        dict(kind="gradient", name="gradient-polymer-80A", material="lamellar", x=80.0, y=61.0,
             z=77.0, r=0.35, dq=0.05, max_q=2.2, slices=150, deposit="nearest", sigma=1.7,
             pixels=257, psis=31, psi_end=90.0, checkpoint=16),
    ]


def draw(rng):
    def spread(lo, hi):
        return math.exp(rng.uniform(math.log(lo), math.log(hi)))

    def box(lo, hi):
        e = spread(lo, hi)
        return dict(zip("xyz", (round(min(hi, e * rng.uniform(0.7, 1.3)), 1) for _ in range(3))))

    def resolution(edge, q_hi=4.0):
        """r, dq and max_q that a slab of this edge allows, the crop at most
        that of the largest listed case."""
        r = round(rng.uniform(0.22, 0.5), 3)
        dq = round(2 * math.pi / (edge * rng.uniform(1.6, 3.5)), 4)
        dq = min(max(dq, 0.02), 0.15)
        top = min(q_hi, 200 * dq, 0.9 * (math.pi / r) / math.sqrt(2) - 6 * dq)
        return dict(r=r, dq=dq, max_q=round(rng.uniform(0.6, 1.0) * top, 2))

    kind = rng.choice(["voxel", "voxel", "voxel", "detector", "simulate", "fit", "gradient"])
    if kind == "voxel":
        material = rng.choice(["graphite", "silicon", "occupied", "lamellar"])
        n = rng.choice([1, 1, 1, int(spread(2, 12))])
        b = box(12, 110 if n == 1 else 60)
        return dict(VOXEL, material=material, **b, **resolution(max(b.values())),
                    slices=int(spread(20, 400 if n == 1 else 180)), structures=n,
                    fill=rng.random() < 0.4, smooth=rng.choice([0.0, 1.0, 1.5, 2.0]),
                    accum=rng.choice(["fp64", "fp64", "fp64", "kahan32"]))
    if kind == "detector":
        general = rng.random() < 0.5
        dq = round(rng.uniform(0.02, 0.08), 3)
        return dict(DETECTOR, r=0.3, dq=dq, max_q=round(rng.uniform(0.5, 1.0) * min(3.5, 180 * dq), 2),
                    pixels=int(spread(64, 1000 if not general else 500)),
                    psis=int(spread(4, 181)) if not general else rng.randint(1, 12),
                    psi_end=round(rng.uniform(10, 180), 1), init_psi=rng.choice([0.0, 90.0]),
                    phis=rng.randint(3, 90) if general else 1, phi_end=170.0,
                    thetas=rng.choice([1, 2]) if general else 1, theta_end=12.5,
                    mirror=rng.random() < 0.7)
    image = dict(pixels=int(spread(64, 800)), psis=int(spread(4, 120)), psi_end=90.0)
    if kind == "simulate":
        b = box(12, 90)
        return dict(SIMULATE, material=rng.choice(["graphite", "silicon", "lamellar"]), **b,
                    **resolution(max(b.values()), 3.0), slices=int(spread(20, 300)),
                    fill=rng.random() < 0.5, smooth=rng.choice([0.0, 1.0, 2.0]),
                    init_psi=rng.choice([0.0, 90.0]), **image)
    if kind == "fit":
        size = round(spread(20, 60), 1)
        return dict(kind="fit", **resolution(1.3 * size, 2.5), candidates=rng.randint(1, 9), size=size,
                    slices=int(spread(20, 180)), smooth=rng.choice([0.0, 1.0]),
                    **dict(image, pixels=min(400, image["pixels"])))
    b = box(14, 70)
    return dict(kind="gradient", material=rng.choice(["silicon", "lamellar"]), **b,
                **resolution(max(b.values()), 3.0), slices=int(spread(20, 180)),
                deposit=rng.choice(["nearest", "bilinear"]),
                # clear of whole numbers, where the plateau's edge jumps
                sigma=round(rng.randint(1, 2) + rng.uniform(0.2, 0.8), 2),
                **dict(image, pixels=min(512, image["pixels"])), checkpoint=16)


# ------------------------------------------------------------------ inputs
def _structure(case, rng, size=None):
    """(coords (N, 3), elements (N,), weights (N,) or None) of a slab."""
    from giwaxsim_gb300 import workloads as W
    size = np.array([case["x"], case["y"], case["z"]] if size is None else size)
    if case["material"] == "lamellar":
        xyz, el = W.lamellar_slab(float(size.max()), rng)
        keep = np.all(xyz < size, axis=1)
        return np.ascontiguousarray(xyz[keep]), el[keep], None
    if case["material"] == "graphite":
        xyz, e = W.graphite_slab(size, rng, disp_sigma=0.1, vacancy=0.05)
    else:
        xyz, e = W.silicon_slab(size, rng, disp_sigma=0.08)
    w = rng.uniform(0.8, 1.0, len(xyz)) if case["material"] == "occupied" else None
    return xyz, np.full(len(xyz), e), w


def _structures(case, seed):
    rng = np.random.default_rng(seed)
    n = case.get("structures", 1)
    box = np.array([case["x"], case["y"], case["z"]])
    out = []
    for _ in range(n):
        out.append(_structure(case, rng, box * rng.uniform(0.4, 1.6, 3) if n > 1 else box))
    return out


def _f_values(elements, weights=None):
    kinds = np.unique(elements)
    f = np.zeros(len(elements), complex)
    for e in kinds:
        f[elements == e] = Z[str(e)] + F1F2[str(e)]
    return f if weights is None else f * weights


def _phis(case):
    n = case["slices"]
    return np.linspace(0.0, 180.0 - 180.0 / n, n)


def _angles(case):
    """psi, phi and theta lists of the detector sum."""
    psis = np.linspace(0.0, case["psi_end"], case["psis"])
    phis = np.linspace(0.0, case.get("phi_end", 0.0), case.get("phis", 1))
    thetas = np.linspace(0.0, case.get("theta_end", 0.0), case.get("thetas", 1))
    return psis, phis, thetas


def _init(case):
    p = case.get("init_psi", 0.0)
    return (p, 0.0, 0.0), (("psi" if p else "None"), "None", "None")


def _speckle(case, seed):
    """An I(q) of the kind the voxel stage makes: speckle (an exponential
    distribution) under a falling envelope, on the cropped cube."""
    g, q, lo, hi = _axes(case["r"], case["dq"], case["max_q"])
    qc = q[lo:hi + 1]
    rng = np.random.default_rng(seed)
    iq = rng.standard_exponential((len(qc),) * 3, dtype=np.float32).astype(np.float64)
    fall = np.exp(-0.5 * (qc / case["max_q"]) ** 2)
    iq *= 1e4 * fall[:, None, None]
    iq *= (fall[:, None] * fall[None, :])[None]
    return iq, qc


def _target(case, seed):
    """A measured pattern: rings of some width on a falling background."""
    rng = np.random.default_rng(seed + 1)
    h = np.linspace(-case["max_q"], case["max_q"], case["pixels"])
    q = np.hypot(h[:, None], h[None, :])
    img = 0.05 * np.exp(-q)
    for _ in range(12):
        img += rng.uniform(0.2, 1.0) * np.exp(-((q - rng.uniform(0.3, 1.2) * case["max_q"]) / 0.08) ** 2)
    return img * rng.uniform(0.95, 1.05, img.shape)


def _sizes(case, seed):
    """The candidates of a search round: sizes along the diagonal around a
    start."""
    s = case["size"] * np.random.default_rng(seed).uniform(0.92, 1.08, 3)
    return [tuple(float(v) for v in s * c) for c in np.linspace(0.85, 1.15, case["candidates"])]


class _DeviceIq:
    """The float32 I(q) a plan keeps on the device, for torch.as_tensor (the
    tensor holds this object, and it the plan, whose memory it is)."""

    def __init__(self, plan):
        self.plan = plan
        self.__cuda_array_interface__ = dict(shape=(plan.Qc,) * 3, typestr="<f4", version=3,
                                             data=(plan.device_iq32(), False))


def prepare(case, seed):
    return globals()["_prepare_" + case["kind"]](case, seed)


def run(state):
    return state["run"](state)


def _prepare_voxel(case, seed):
    from giwaxsim_gb300.forward import VoxelGeometry, VoxelPlan
    items = [(xyz, _f_values(el), w) for xyz, el, w in _structures(case, seed)]
    plan = VoxelPlan(VoxelGeometry(case["r"], case["dq"], case["max_q"]), items, phis=_phis(case),
                     fill_bkg=case["fill"], smooth=case["smooth"], accum=case["accum"])
    xyz = torch.as_tensor(plan.xyz).cuda()
    f = torch.as_tensor(plan.f).cuda()
    torch.cuda.synchronize()
    plan.set_atoms(xyz.data_ptr(), f.data_ptr(), on_device=True)
    plan.capture_graph()
    iq = torch.as_tensor(_DeviceIq(plan), device="cuda")
    return dict(run=_run_voxel, plan=plan, xyz=xyz, f=f, iq=iq)


def _run_voxel(s):
    s["plan"].set_atoms(s["xyz"].data_ptr(), s["f"].data_ptr(), on_device=True)
    s["plan"].execute()
    return s["iq"]


def _detector_args(case):
    psis, phis, thetas = _angles(case)
    vals, axs = _init(case)
    return case["pixels"], case["max_q"], vals, axs, psis, None, phis, None, thetas, None


def _prepare_detector(case, seed):
    iq, q = _speckle(case, seed)
    return dict(run=_run_detector, iq=iq, q=q, args=_detector_args(case), mirror=case["mirror"])


def _run_detector(s):
    from giwaxsim_gb300.tools.comparison import detectormaker_fitting
    image, _, _ = detectormaker_fitting(s["iq"], s["q"], s["q"], s["q"], *s["args"], mirror=s["mirror"])
    return image


def _prepare_simulate(case, seed):
    (xyz, el, _), = _structures(case, seed)
    return dict(run=_run_simulate, case=case, xyz=xyz, el=el, phis=_phis(case), args=_detector_args(case))


def _run_simulate(s):
    from giwaxsim_gb300.tools.comparison import detectormaker_fitting, voxelgridmaker_fitting
    c = s["case"]
    iq, qx, qy, qz = voxelgridmaker_fitting(s["xyz"], s["el"], c["r"], c["dq"], c["max_q"], ENERGY,
                                            fill_bkg=c["fill"], smooth=c["smooth"], phis=s["phis"],
                                            f1f2=F1F2)
    image, _, _ = detectormaker_fitting(iq, qx, qy, qz, *s["args"], mirror=True)
    return image.astype(np.float32)


def _prepare_fit(case, seed):
    from giwaxsim_gb300 import workloads as W
    from giwaxsim_gb300.fit import SlabFit
    cell = W.GRAPHITE_BASIS @ W.GRAPHITE_CELL
    t = np.linspace(0.0, case["max_q"], 33)
    fit = SlabFit(cell, ["C"] * 4, GRAPHITE, case["r"], case["dq"], case["max_q"], ENERGY,
                  case["pixels"], np.ones((33, 33)), t, t, np.zeros((33, 33)), smooth=case["smooth"],
                  phis=_phis(case), psis=_angles(case)[0], f1f2=F1F2)
    return dict(run=_run_fit, fit=fit, sizes=_sizes(case, seed))


def _run_fit(s):
    return np.stack(s["fit"].images(s["sizes"])).astype(np.float32)


def _parameters(case, seed):
    """Occupancies, sigma and coordinates at the start of a refinement, in
    float32, and the elements: one model of the case's slab (its atoms are
    the same ones for every seed), displaced."""
    (xyz, el, _), = _structures(case, 5)
    rng = np.random.default_rng(seed)
    xyz = xyz + rng.normal(0.0, 0.05, xyz.shape)
    occ = rng.uniform(0.7, 1.0, len(xyz))
    return occ.astype(np.float32), np.float32(case["sigma"]), xyz.astype(np.float32), el


def _prepare_gradient(case, seed):
    from giwaxsim_gb300.autograd import DetectorModel
    occ, sigma, xyz, el = _parameters(case, seed)
    model = DetectorModel(el, ENERGY, case["r"], case["dq"], case["max_q"], case["pixels"],
                          psis=_angles(case)[0], phis=_phis(case), deposit=case["deposit"],
                          checkpoint_every=case["checkpoint"], f1f2=F1F2)
    bilinear = case["deposit"] == "bilinear"
    return dict(run=_run_gradient, model=model, target=torch.as_tensor(_target(case, seed)),
                occ=torch.tensor(occ, requires_grad=True), sigma=torch.tensor(sigma, requires_grad=True),
                xyz=torch.tensor(xyz, requires_grad=bilinear))


def _run_gradient(s):
    from giwaxsim_gb300.autograd import detector_image, scale_offset_misfit
    params = [s["occ"], s["sigma"], s["xyz"]]
    for p in params:
        p.grad = None
    image = detector_image(s["model"], *params)
    loss, _, _ = scale_offset_misfit(image, s["target"])
    loss.backward()
    return [p.grad for p in params if p.requires_grad]


# ------------------------------------------------------------------ work
def _voxel_work(case, n_struct=1, real=True, edges=None):
    """Bytes and operations of the voxel stage: atoms in, float32 I(q) out;
    per slice the two 1-D transforms of the slab's footprint to the band that
    lands in the crop, as FFTs of the longer of the two."""
    x, y, z = edges or (case["x"], case["y"], case["z"])
    g, q, lo, hi = _axes(case["r"], case["dq"], case["max_q"])
    n = hi - lo + 1
    atoms = n_struct * x * y * z * (0.113 if case.get("material", "graphite") == "graphite" else
                                    0.05 if case["material"] != "lamellar" else 0.033)
    ly, lz = math.hypot(x, y) / case["r"], z / case["r"]
    nz = 2 * case["max_q"] * g * case["r"] / (2 * math.pi)
    ny = nz * 1.2
    fft = lambda m: 5 * m * math.log2(m)  # noqa: E731
    ops = lz * fft(max(ly, ny, 2)) + ny * fft(max(lz, nz, 2))
    flops = n_struct * case["slices"] * ops * (0.5 if real else 1.0)
    return 32 * atoms + 4 * n ** 3, flops


def _detector_work(case):
    psis, phis, thetas = _angles(case)
    samples = case["pixels"] ** 2 * len(psis) * len(phis) * len(thetas)
    # one affine map of three coordinates and one weighted add per sample
    return 8 * case["pixels"] ** 2, 20 * samples


def work(case):
    kind = case["kind"]
    if kind == "detector":
        b, f = _detector_work(case)
        g, q, lo, hi = _axes(case["r"], case["dq"], case["max_q"])
        n = hi - lo + 1
        plane = len(_angles(case)[1]) == 1 and len(_angles(case)[2]) == 1
        return dict(bytes=b + 8 * (n * n if plane else n ** 3), flops=f)
    real = case.get("material") != "lamellar"
    if kind == "voxel":
        b, f = _voxel_work(case, case["structures"], real)
        return dict(bytes=b, flops=f)
    if kind == "simulate":
        (b, f), (b2, f2) = _voxel_work(case, 1, real), _detector_work(case)
        return dict(bytes=b + b2, flops=f + f2)
    if kind == "fit":
        k = case["candidates"]
        (b, f), (b2, f2) = _voxel_work(case, 1, True, (case["size"],) * 3), _detector_work(case)
        return dict(bytes=k * (b + b2), flops=k * (f + f2))
    # a gradient: the forward, and about twice it backwards
    (b, f), (b2, f2) = _voxel_work(case, 1, False), _detector_work(case)
    return dict(bytes=2 * (b + b2), flops=3 * (f + f2))


# ------------------------------------------------------------------ exact
def _axes(r, dq, max_q):
    """Grid size, q axis and crop range, as numpy's float64 gives them."""
    diag = np.sqrt(2) * max_q
    g = int(np.ceil(2 * np.pi / (dq * r)))
    diag = diag + diag % dq
    n = int(2 * diag / dq + 1)
    n += n % 2 == 0
    q = np.linspace(-diag, diag, n)
    keep = np.where(np.abs(q) < max_q + np.abs(q[1] - q[0]))[0]
    return g, q, int(keep[0]), int(keep[-1])


def _fma(a, b, c):
    """a b + c rounded once (numpy or torch float64): the product by
    Dekker's splitting, the sum with its error term."""
    p = a * b
    t = 134217729.0 * a
    ah = t - (t - a)
    t = 134217729.0 * b
    bh = t - (t - b)
    e = ((ah * bh - p) + ah * (b - bh) + (a - ah) * bh) + (a - ah) * (b - bh)
    s = p + c
    v = s - p
    return s + (((p - (s - v)) + (c - v)) + e)


def _floor_div(a, b):
    """numpy's float64 a // b for b > 0: the exact floor."""
    k = torch.floor(a / b)
    k = torch.where(_fma(-k, torch.full_like(k, b), a) < 0, k - 1, k)
    return torch.where(_fma(-(k + 1), torch.full_like(k, b), a) >= 0, k + 1, k)


def _rotate(R, p):
    """R p, each row the fused chain of a BLAS product."""
    return tuple(_fma(p[2], p[2] * 0 + R[i, 2], _fma(p[1], p[1] * 0 + R[i, 1], p[0] * R[i, 0]))
                 for i in range(3))


def _collapse(x, hor, ver, phi):
    """Path length through a hor x ver rectangle turned by phi, per column."""
    if phi > 90:
        phi, hor, ver = phi - 90, ver, hor
    if phi == 0:
        return np.where(x < hor, ver, 0.0)
    if phi == 90:
        return np.where(x < ver, hor, 0.0)
    t, p = np.deg2rad(90 - phi), np.deg2rad(phi)
    vc = ver * np.cos(t)
    s1, s2 = vc, hor * np.cos(p)
    if s1 < s2:
        mid = ver / np.sin(t)
    else:
        s1, s2 = s2, s1
        mid = hor / np.sin(p)
    base = np.sqrt(ver ** 2 - vc ** 2)
    rise = (base + x * np.tan(p)) - ((vc - x) * np.tan(t))
    fall = (hor - ((x - vc) / np.cos(p))) / np.cos(t)
    out = np.where(x < s1, rise, np.where(x <= s2, mid, np.where(x < s1 + s2, fall, 0.0)))
    return np.where(x == 0, 0.0, out)


def _profile(g, lo, hi, sigma):
    """The plateau [lo + sigma, hi - sigma) under a wrapped Gaussian filter
    cut at four sigma; sigma a tensor."""
    v = float(sigma)
    s, e, _ = slice(int(math.ceil(lo + v)), int(math.ceil(hi - v))).indices(g)
    radius = int(4.0 * v + 0.5)
    j = torch.arange(-radius, radius + 1, dtype=torch.float64, device="cuda")
    w = torch.exp(-0.5 * j * j / (sigma * sigma))
    w = w / w.sum()
    at = (torch.arange(g, device="cuda")[:, None] + torch.arange(-radius, radius + 1, device="cuda")) % g
    return (((at >= s) & (at < e)).double() * w).sum(1)


def _dense_sum(xyz, f, case, phis, fill, sigma, deposit="nearest"):
    """Binned |F|^2 of one structure over all slices (Qc^3, on the GPU) as a
    differentiable function of f, xyz and sigma (tensors), and the counts."""
    r = case["r"]
    g, q, lo, hi = _axes(r, case["dq"], case["max_q"])
    n = hi - lo + 1
    ext = xyz.amax(0) - xyz.amin(0)
    avg = f.sum() / (ext[0] * ext[1] * ext[2]) * r ** 3
    xb, yb = float(ext[0]), float(ext[1])
    depth = float(np.sqrt(xb ** 2 + yb ** 2) // r)
    c = avg * depth
    pos = xyz.detach()
    zv = pos[:, 2] - pos[:, 2].min()
    zi = _floor_div(zv, r).long()
    h_max = np.max(np.fft.fftfreq(g, d=r) * 2 * np.pi)
    qv = np.fft.fftshift(np.fft.fftfreq(g, d=r) * 2 * np.pi)
    step = np.diff(q)[0]
    total = torch.zeros(n ** 3, dtype=torch.float64, device="cuda")
    c2, c1 = np.zeros(n * n), np.zeros(n)
    rows = np.where((qv <= np.max(q)) & (qv >= np.min(q)))[0]
    iz = ((qv[rows] - np.min(q)) // step).astype(int) - lo
    rows, iz = rows[(iz >= 0) & (iz < n)], iz[(iz >= 0) & (iz < n)]
    np.add.at(c1, iz, 1.0)
    iz = torch.as_tensor(iz, device="cuda")
    rows = torch.as_tensor((rows - g // 2) % g, device="cuda")
    for phi in phis:
        pr = np.radians(phi)
        sn, cs = float(np.sin(pr)), float(np.cos(pr))
        y = _fma(pos[:, 1], torch.full_like(pos[:, 1], cs), pos[:, 0] * sn)
        yi = _floor_div(y - y.min(), r).long()
        ok = (yi < g) & (zi < g)
        yk, zk, fk = yi[ok], zi[ok], f[ok]
        if deposit == "nearest":
            cells, vals = zk * g + yk, fk
        else:
            yt = xyz[:, 0] * sn + xyz[:, 1] * cs
            fu = ((yt - yt.min()) / r - yi)[ok]
            fz = ((xyz[:, 2] - xyz[:, 2].min()) / r - zi)[ok]
            cells, vals = [], []
            for dz in (0, 1):
                for dy in (0, 1):
                    m = (zk + dz < g) & (yk + dy < g)
                    cells.append(((zk + dz) * g + yk + dy)[m])
                    vals.append((fk * ((fz if dz else 1 - fz) * (fu if dy else 1 - fu)))[m])
            cells, vals = torch.cat(cells), torch.cat(vals)
        grid = torch.zeros(g * g, 2, dtype=torch.float64, device="cuda").index_add(
            0, cells, torch.view_as_real(vals))
        grid = torch.view_as_complex(grid).view(g, g)
        y0, y1, z0, z1 = (int(v) for v in (yk.min(), yk.max(), zk.min(), zk.max()))
        if fill:
            lens = _collapse(np.arange(g) * r, yb, xb, phi)
            missing = torch.as_tensor((depth - lens // r).astype(int), device="cuda")
            grid = grid + (missing * avg)[None, :]
            grid[:z0] = c
            grid[z1:] = c
            grid[z0:z1 + 1, :y0 + 1] = c
            grid[z0:z1 + 1, y1:] = c
        if float(sigma) > 0:
            m = _profile(g, z0, z1, sigma)[:, None] * _profile(g, y0, y1, sigma)[None, :]
            grid = grid * m + c * (1 - m)
        hy = np.linspace(-h_max * np.cos(np.deg2rad(-phi)), h_max * np.cos(np.deg2rad(-phi)), num=g)
        hx = np.linspace(h_max * np.sin(np.deg2rad(-phi)), -h_max * np.sin(np.deg2rad(-phi)), num=g)
        cols = np.where((hx <= np.max(q)) & (hx >= np.min(q)) & (hy <= np.max(q)) & (hy >= np.min(q)))[0]
        ix = ((hx[cols] - np.min(q)) // step).astype(int) - lo
        iy = ((hy[cols] - np.min(q)) // step).astype(int) - lo
        m = (ix >= 0) & (ix < n) & (iy >= 0) & (iy < n)
        line = iy[m] * n + ix[m]
        np.add.at(c2, line, 1.0)
        cols = torch.as_tensor((cols[m] - g // 2) % g, device="cuda")
        line = torch.as_tensor(line, device="cuda")
        F = torch.fft.fft(torch.fft.fft(grid, dim=0)[rows], dim=1)[:, cols]
        I = F.real ** 2 + F.imag ** 2
        total = total.index_add(0, (line[None, :] * n + iz[:, None]).reshape(-1), I.reshape(-1))
    return total, c2, c1


def _dense_iq(structs, case, phis, fill, sigma, deposit="nearest"):
    """I(q) averaged over structures [(xyz, f)], divided by the counts, with
    carbon's f0 squared."""
    total = 0.0
    for xyz, f in structs:
        s, c2, c1 = _dense_sum(xyz, f, case, phis, fill, sigma, deposit)
        total = total + s
    g, q, lo, hi = _axes(case["r"], case["dq"], case["max_q"])
    n = hi - lo + 1
    q2 = torch.as_tensor(q[lo:hi + 1] ** 2, device="cuda")
    q2 = (q2[None, :, None] + q2[:, None, None] + q2[None, None, :]).reshape(-1) / (16 * np.pi ** 2)
    f0 = F0_C[8] + sum(F0_C[2 * i] * torch.exp(-F0_C[2 * i + 1] * q2) for i in range(4))
    del q2
    count = (torch.as_tensor(c2, device="cuda")[:, None] * torch.as_tensor(c1, device="cuda")[None, :]).reshape(-1)
    scale = torch.where(count > 0, (f0 / Z["C"]) ** 2 / count.clamp(min=1), torch.zeros_like(f0))
    return (total * scale / len(structs)).view(n, n, n)


def _turn(axis, angle):
    """The rotation about a unit axis by an angle in degrees."""
    t = np.radians(angle)
    x, y, z = axis
    k = 1 - np.cos(t)
    return np.array([
        [np.cos(t) + x ** 2 * k, x * y * k - z * np.sin(t), x * z * k + y * np.sin(t)],
        [y * x * k + z * np.sin(t), np.cos(t) + y ** 2 * k, y * z * k - x * np.sin(t)],
        [z * x * k - y * np.sin(t), z * y * k + x * np.sin(t), np.cos(t) + z ** 2 * k]])


def _plane_turn(corners, kind, angle):
    """The plane turned about its normal (psi) or one of its edges."""
    p1, p2, p3 = np.stack(corners, 1)
    axis = np.cross(p2 - p1, p3 - p1) if kind == "psi" else p2 - p1 if kind == "theta" else p3 - p1
    return _turn(axis / np.linalg.norm(axis), angle)


def _dense_image(iq, case, mirror=True):
    """The detector image of I(q) (Qc, Qc, Qc; a tensor on the GPU)."""
    g, q, lo, hi = _axes(case["r"], case["dq"], case["max_q"])
    q = q[lo:hi + 1]
    n, step = len(q), float(np.diff(q)[0])
    h = np.linspace(-case["max_q"], case["max_q"], case["pixels"])
    yy, zz = (torch.as_tensor(a.reshape(-1), device="cuda") for a in np.meshgrid(h, h))
    plane = (torch.zeros_like(yy), yy, zz)
    corners = (np.zeros(3), np.array([h[0], h[-1], h[0]]), np.array([h[0], h[0], h[-1]]))
    for val, kind in zip(*_init(case)):
        if kind != "None":
            R = _plane_turn(corners, kind, val)
            plane, corners = _rotate(R, plane), _rotate(R, corners)
    psis, phis, thetas = _angles(case)
    w = 1.0 / len(psis) * (1.0 / len(phis)) * (1.0 / len(thetas))
    flat = iq.reshape(-1)
    total = torch.zeros_like(yy)

    def place(v):
        return _floor_div(v - float(np.min(q)), step).clamp(0, n - 1).long()

    for psi in psis:
        R = _plane_turn(corners, "psi", psi)
        p1, c1 = _rotate(R, plane), _rotate(R, corners)
        for phi in phis:
            R = _plane_turn(c1, "phi", phi)
            p2, c2 = (_rotate(R, p1), _rotate(R, c1)) if phi else (p1, c1)
            for theta in thetas:
                p3 = _rotate(_plane_turn(c2, "theta", theta), p2) if theta else p2
                total = total + w * flat[(place(p3[1]) * n + place(p3[0])) * n + place(p3[2])]
    image = total.view(case["pixels"], case["pixels"])
    if mirror:
        image = image + image.flip(1) + image.flip(0) + image.flip(0).flip(1)
    return torch.where(image > 0, image, torch.full_like(image, 1e-6)) * 1e-6


def _slab(cell, vecs, size):
    """A cell tiled over a box twice the size and cut to its middle."""
    a, b, c = vecs
    xyz = np.array(cell)
    for k, v in enumerate((a, b, c)):
        reps = int(np.ceil(2 * size[k] / v[k]))
        xyz = np.concatenate([xyz] + [xyz + v * (i + 1) for i in range(reps)])
    ext = xyz.max(0) - xyz.min(0)
    margin = (ext - np.array(size)) / 2
    xyz = xyz - xyz.min(0)
    xyz = xyz[np.all((xyz >= margin) & (xyz <= ext - margin), axis=1)]
    return xyz - xyz.min(0)


def _gpu(xyz, f):
    return torch.as_tensor(np.asarray(xyz, np.float64)).cuda(), torch.as_tensor(f).cuda()


def exact(case, seed):
    kind = case["kind"]
    if kind == "detector":
        iq, _ = _speckle(case, seed)
        return _dense_image(torch.as_tensor(iq).cuda(), case, case["mirror"]).cpu().numpy()
    if kind == "gradient":
        return _exact_gradient(case, seed)
    phis = _phis(case)
    sigma = torch.tensor(float(case["smooth"]), dtype=torch.float64, device="cuda")
    with torch.no_grad():
        if kind == "fit":
            from giwaxsim_gb300 import workloads as W
            cell = W.GRAPHITE_BASIS @ W.GRAPHITE_CELL
            a, _, c, _, _, gamma = GRAPHITE
            ga = np.deg2rad(gamma)
            right = np.cos(np.deg2rad(90.0))
            vc = [a * 0 + c * right, c * (right - right * np.cos(ga)) / np.sin(ga)]
            vol = a * a * c * np.sqrt(1 - right ** 2 - right ** 2 - np.cos(ga) ** 2 + 2 * right * right * np.cos(ga))
            vecs = (np.array([a, 0, 0]), np.array([a * np.cos(ga), a * np.sin(ga), 0]),
                    np.array([vc[0], vc[1], vol / (a * a * np.sin(ga))]))
            out = []
            for size in _sizes(case, seed):
                xyz = _slab(cell, vecs, size)
                s = [_gpu(xyz, _f_values(np.full(len(xyz), "C")))]
                out.append(_dense_image(_dense_iq(s, case, phis, False, sigma), case).cpu().numpy())
            return np.stack(out)
        structs = [_gpu(xyz, _f_values(el, w)) for xyz, el, w in _structures(case, seed)]
        iq = _dense_iq(structs, case, phis, case["fill"], sigma)
        return iq if kind == "voxel" else _dense_image(iq, case).cpu().numpy()


def _exact_gradient(case, seed):
    occ, sigma, xyz, el = _parameters(case, seed)
    bilinear = case["deposit"] == "bilinear"
    o, s, x = (torch.tensor(np.asarray(v, np.float64), device="cuda", requires_grad=g)
               for v, g in ((occ, True), (sigma, True), (xyz, bilinear)))
    f = torch.as_tensor(_f_values(el)).cuda() * o
    phis = _phis(case)
    # the slices in groups: first I(q) alone, then the groups again with the
    # gradient of the misfit by I(q) in hand
    with torch.no_grad():
        iq = _dense_iq([(x, f)], case, phis, False, s, case["deposit"])
        ones, c2, c1 = _dense_sum(x, f, case, phis, False, s, case["deposit"])
    iq.requires_grad_(True)
    image, target = _dense_image(iq, case).reshape(-1), torch.as_tensor(_target(case, seed)).cuda().reshape(-1)
    n = image.numel()
    det = n * (image * image).sum() - image.sum() ** 2
    scale = (n * (image * target).sum() - image.sum() * target.sum()) / det
    offset = (target.sum() - scale * image.sum()) / n
    g_iq, = torch.autograd.grad(((scale * image + offset - target) ** 2).sum(), iq)
    with torch.no_grad():  # dI/dsum
        per_sum = torch.where(ones > 0, iq.reshape(-1) / ones, torch.zeros_like(ones))
    g_sum = g_iq.reshape(-1) * per_sum
    for k in range(0, len(phis), 16):
        f = torch.as_tensor(_f_values(el)).cuda() * o
        part, _, _ = _dense_sum(x, f, case, phis[k:k + 16], False, s, case["deposit"])
        (part * g_sum).sum().backward()
    return [p.grad for p in (o, s, x) if p.requires_grad]
