"""Performance cases of the library: the calls a registration program makes, from one objective
evaluation of a small volume to whole registrations and a full-size CT gradient.

A case names its `kind` (the public entry point or sequence of them) and its sizes:

    objective  one fused objective evaluation          (nrb.f3d_objective)
    gradient   one fused gradient evaluation           (nrb.f3d_gradient)
    steps      one iteration call by call, as a platform binding drives it: field, warp, NMI,
               bending energy, spatial and voxel gradients, nodes, conjugate gradient, update
    warp       the final warped image                  (nrb.f3d_warped_image)
    velocity   a velocity grid exponentiated           (nrb.get_def_field_from_velocity_grid)
    pyramid    an image pyramid and the finest level's intensity rescale
    register   a whole registration, device images     (nrb.register_device)
    batch      many small registrations, host images   (nrb.register_batch)
    f3d2       a symmetric registration, host images   (nrb.f3d2_register_images)

Volumes are [nz, ny, nx] float32, x fastest; inputs are seeded phantoms (a head of labelled
ellipsoids with noise and a bias field; the floating image warped by a random free-form
deformation), made on the GPU. `exact` restates each evaluation in 64-bit torch.
"""
import math

import numpy as np
import torch

import niftyreg_b200 as nrb

BE = 0.005  # bending-energy weight of the repository's benchmark configurations
MARGIN_BINS = 4  # the Parzen margin added to the user's bin count


def listed():
    return [
        # one line-search evaluation of a small volume (the coarse levels of every registration)
        {"name": "objective_64", "kind": "objective", "nx": 64, "ny": 64, "nz": 64, "spacing": 5.0, "bins": 64,
         "px": 1.0, "pz": 1.0},
        # one line-search evaluation of the benchmark's brain volume
        {"name": "objective_brain", "kind": "objective", "nx": 182, "ny": 218, "nz": 182, "spacing": 5.0, "bins": 64,
         "px": 1.0, "pz": 1.0},
        # one gradient evaluation of the same
        {"name": "gradient_brain", "kind": "gradient", "nx": 182, "ny": 218, "nz": 182, "spacing": 5.0, "bins": 64,
         "px": 1.0, "pz": 1.0},
        # the largest configuration: CT volume, 128 bins, anisotropic voxels, 10 mm grid
        {"name": "gradient_ct", "kind": "gradient", "nx": 512, "ny": 512, "nz": 320, "spacing": 10.0, "bins": 128,
         "px": 0.8, "pz": 1.5},
        # an iteration of NiftyReg's own driver on the call-by-call interface: odd dims, a mask
        {"name": "steps_odd", "kind": "steps", "nx": 181, "ny": 217, "nz": 181, "spacing": 5.0, "bins": 64,
         "px": 1.0, "pz": 1.0, "mask": True},
        # the image a registration delivers: cubic-spline warp of the floating volume
        {"name": "warp_brain", "kind": "warp", "nx": 182, "ny": 218, "nz": 182, "spacing": 5.0, "order": 3,
         "px": 1.0, "pz": 1.0},
        # F3D2: one exponentiation of a velocity grid over the brain volume
        {"name": "velocity_brain", "kind": "velocity", "nx": 182, "ny": 218, "nz": 182, "spacing": 5.0,
         "px": 1.0, "pz": 1.0},
        # preparing a CT volume: three pyramid levels and the intensity rescale
        {"name": "pyramid_ct", "kind": "pyramid", "nx": 512, "ny": 512, "nz": 320, "levels": 3, "bins": 128,
         "px": 0.8, "pz": 1.5},
        # a small registration (config: 64^3, one level, 100 iterations)
        {"name": "register_64", "kind": "register", "nx": 64, "ny": 64, "nz": 64, "spacing": 5.0, "bins": 64,
         "px": 1.0, "pz": 1.0, "levels": 1, "iterations": 100},
        # the headline registration: brain volume, three levels, 300 iterations
        {"name": "register_brain", "kind": "register", "nx": 182, "ny": 218, "nz": 182, "spacing": 5.0, "bins": 64,
         "px": 1.0, "pz": 1.0, "levels": 3, "iterations": 300},
        # a cohort of small and medium pairs in one batch
        {"name": "batch_16", "kind": "batch", "nx": 96, "ny": 96, "nz": 80, "spacing": 5.0, "bins": 64,
         "px": 1.0, "pz": 1.0, "levels": 2, "iterations": 50, "pairs": 16},
        # a symmetric registration of an obliquely scanned pair
        {"name": "f3d2_oblique", "kind": "f3d2", "nx": 96, "ny": 112, "nz": 88, "spacing": 5.0, "bins": 64,
         "px": 1.0, "pz": 1.1, "levels": 2, "iterations": 20, "oblique": True},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["objective", "objective", "gradient", "gradient", "steps", "warp", "velocity", "pyramid",
                       "register", "batch", "f3d2"])
    # a size per axis: edge lengths around a drawn scale, odd ones as often as even ones
    top = {"objective": 400, "gradient": 320, "steps": 240, "warp": 256, "velocity": 220, "pyramid": 384,
           "register": 160, "batch": 88, "f3d2": 96}[kind]
    edge = _log_int(rng, 40, top)
    dims = [max(24, int(edge * rng.uniform(0.8, 1.2))) for _ in range(3)]
    c = {"kind": kind, "nx": dims[0], "ny": dims[1], "nz": dims[2], "px": rng.choice([0.8, 1.0, 1.0, 1.2]),
         "pz": rng.choice([1.0, 1.0, 1.5, 2.0])}
    if kind != "pyramid":
        c["spacing"] = rng.choice([5.0, 5.0, 6.0, 8.0, 10.0])
    if kind not in ("warp", "velocity"):
        c["bins"] = rng.choice([32, 64, 64, 128]) if kind not in ("register", "batch", "f3d2") else 64
    if kind in ("objective", "gradient", "steps"):
        c["mask"] = rng.random() < 0.3
    if kind == "warp":
        c["order"] = rng.choice([0, 1, 3, 3])
    if kind == "velocity":
        c["oblique"] = rng.random() < 0.3
    if kind == "pyramid":
        c["levels"] = rng.choice([2, 3])
    if kind in ("register", "batch", "f3d2"):
        c["levels"] = rng.choice([1, 2])
        c["iterations"] = rng.choice([10, 20, 30])
    if kind == "batch":
        c["pairs"] = rng.choice([3, 6, 11])
    if kind == "f3d2":
        c["oblique"] = rng.random() < 0.5
    return c


# ------------------------------------------------------------------------------------------------
# seeded inputs
# ------------------------------------------------------------------------------------------------
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _axes(shape):
    nz, ny, nx = shape
    z = torch.arange(nz, device="cuda", dtype=torch.float32).view(nz, 1, 1)
    y = torch.arange(ny, device="cuda", dtype=torch.float32).view(1, ny, 1)
    x = torch.arange(nx, device="cuda", dtype=torch.float32).view(1, 1, nx)
    return z, y, x


def _head(shape, gen, seed):
    """Labelled phantom: class means 250/500/750 in a head ellipsoid, noise, a bias field."""
    r = np.random.default_rng(seed)
    nz, ny, nx = shape
    z, y, x = _axes(shape)
    d = lambda c, s: ((z - c[0]) / s[0]) ** 2 + ((y - c[1]) / s[1]) ** 2 + ((x - c[2]) / s[2]) ** 2  # noqa: E731
    n = np.array([nz, ny, nx], float)
    head = d(n / 2, 0.45 * n) <= 1.0
    img = torch.where(head, 250.0, 0.0)
    for _ in range(16):
        c, s, m = n * r.uniform(0.25, 0.75, 3), n * r.uniform(0.05, 0.2, 3), 250.0 * r.integers(1, 4)
        img = torch.where((d(c, s) <= 1.0) & head, torch.full_like(img, m), img)
    noise = torch.empty(shape, device="cuda").normal_(0.0, 30.0, generator=gen)
    img = img + torch.where(head, noise, torch.zeros_like(noise))
    return img * (1.0 + 0.1 * torch.cos(math.pi * z / nz + 0.3) * torch.cos(math.pi * y / ny) * torch.cos(math.pi * x / nx))


def _warped(img, gen, mm, pix):
    """The volume under a smooth random displacement of about `mm` mm."""
    nz, ny, nx = img.shape
    coarse = torch.empty((1, 3, max(4, nz // 12), max(4, ny // 12), max(4, nx // 12)), device="cuda").normal_(generator=gen)
    disp = torch.nn.functional.interpolate(coarse, size=(nz, ny, nx), mode="trilinear", align_corners=True)[0] * mm
    z, y, x = _axes(img.shape)
    grid = torch.stack([2 * (x + disp[0] / pix[0]) / (nx - 1) - 1, 2 * (y + disp[1] / pix[1]) / (ny - 1) - 1,
                        2 * (z + disp[2] / pix[2]) / (nz - 1) - 1], -1)
    return torch.nn.functional.grid_sample(img[None, None], grid[None], mode="bilinear", align_corners=True)[0, 0]


def _pair(case, seed):
    shape = (case["nz"], case["ny"], case["nx"])
    gen = _gen(seed)
    ref = _head(shape, gen, seed)
    return ref, _warped(ref, gen, 3.0, _pix(case))


def _pix(case):
    return (case["px"], case["px"], case["pz"])


def _dim(case):
    return (case["nx"], case["ny"], case["nz"])


def _to_bins(img, bins):
    """Intensities in [2, bins + 1]: what an NMI evaluation with the Parzen margin works on."""
    d = img.double()
    lo, hi = d.min(), d.max()
    return ((d - lo) / (hi - lo) * (bins - 1.0) + 2.0).float().contiguous()


def _rotation(case):
    """Voxel -> mm of an oblique acquisition (small rotations about two axes) or a plain one."""
    m = np.eye(4)
    if case.get("oblique"):
        a, b = 0.12, -0.08
        ra = np.array([[math.cos(a), -math.sin(a), 0], [math.sin(a), math.cos(a), 0], [0, 0, 1]])
        rb = np.array([[1, 0, 0], [0, math.cos(b), -math.sin(b)], [0, math.sin(b), math.cos(b)]])
        m[:3, :3] = ra @ rb
    m[:3, :3] = m[:3, :3] @ np.diag(_pix(case))
    if case.get("oblique"):
        m[:3, 3] = (-30.0, 20.0, 10.0)
    return m.astype(np.float32)


def _geometry(case, xyz=None):
    pix = _pix(case)
    if xyz is None:
        xyz = nrb.identity_header(pix)
    cd, cp, cx = nrb.control_grid_header(_dim(case), pix, (case["spacing"],) * 3)
    if case.get("oblique"):
        # the symmetric grids of F3D2 are axis-aligned in the world: cover the rotated volume
        corners = np.array([[x, y, z, 1.0] for x in (0, case["nx"] - 1) for y in (0, case["ny"] - 1)
                            for z in (0, case["nz"] - 1)]) @ np.asarray(xyz, np.float64).T
        lo, hi = corners[:, :3].min(0), corners[:, :3].max(0)
        s = case["spacing"]
        cd = [int(math.ceil((hi[i] - lo[i]) / s)) + 4 for i in range(3)]
        cx = nrb.identity_header(cp, [float(lo[i] - s) for i in range(3)])
    return nrb.make_geometry(_dim(case), pix, xyz, _dim(case), pix, xyz, cd, cp, cx)


def _grid(g, gen, mm):
    """Control-point positions: the identity grid plus N(0, mm) displacements."""
    cx, cy, cz = list(g.cpp_dim)
    m = torch.tensor(list(g.cpp_xyz), device="cuda").view(4, 4)
    z, y, x = _axes((cz, cy, cx))
    ident = torch.stack([(m[k, 0] * x + m[k, 1] * y + m[k, 2] * z + m[k, 3]).expand(cz, cy, cx) for k in range(3)])
    return (ident + torch.empty_like(ident).normal_(0.0, mm, generator=gen)).contiguous()


def _params(case):
    return nrb.default_params(levels=case["levels"], max_iterations=case["iterations"], bending_energy=BE,
                              spacing=(case["spacing"],), ref_bins=case["bins"], flo_bins=case["bins"])


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case}
    gen = _gen(seed + 1)
    if kind in ("objective", "gradient", "steps"):
        bins = case["bins"]
        ref, flo = _pair(case, seed)
        s["ref"], s["flo"] = _to_bins(ref, bins), _to_bins(flo, bins)
        s["g"] = g = _geometry(case)
        s["cpp"] = _grid(g, gen, 2.0)
        s["ws"], s["nmi"] = nrb.Workspace(g), nrb.Nmi(bins + MARGIN_BINS, bins + MARGIN_BINS)
        s["mask"] = None
        if case.get("mask"):  # the head's bounding region is active
            s["mask"] = torch.where(ref > 100.0, 0, -1).to(torch.int32).contiguous()
        n, nc = g.ref_nvox, g.cpp_nvox
        new = lambda k: torch.zeros(k, device="cuda")  # noqa: E731
        if kind != "objective":
            s["vgrad"], s["node"] = new(3 * n), new(3 * nc)
        if kind == "steps":
            s["def"], s["warped"], s["wgrad"] = new(3 * n), new(n), new(3 * n)
            s["g1"], s["g2"], s["cur"] = new(3 * nc), new(3 * nc), new(3 * nc)
            # the conjugate direction of the previous iteration
            s["g1_0"] = torch.empty(3 * nc, device="cuda").normal_(0.0, 0.3, generator=gen)
            s["g2_0"] = torch.empty(3 * nc, device="cuda").normal_(0.0, 0.3, generator=gen)
    elif kind == "warp":
        s["flo"] = _head((case["nz"], case["ny"], case["nx"]), gen, seed)
        s["g"] = _geometry(case)
        s["cpp"] = _grid(s["g"], gen, 2.0)
        s["warped"] = torch.zeros(s["g"].ref_nvox, device="cuda")
    elif kind == "velocity":
        s["g"] = _geometry(case, _rotation(case))
        s["vel"] = _grid(s["g"], gen, 3.0)
        s["def"] = torch.zeros(3 * s["g"].ref_nvox, device="cuda")
    elif kind == "pyramid":
        s["img"] = _head((case["nz"], case["ny"], case["nx"]), gen, seed)
        s["xyz"] = nrb.identity_header(_pix(case))
        total = nrb.image_pyramid_headers(_dim(case), _pix(case), s["xyz"], case["levels"])[2]
        s["out"] = torch.zeros(total, device="cuda")
        s["finest"] = torch.zeros(s["img"].numel(), device="cuda")
    elif kind == "register":
        ref, flo = _pair(case, seed)
        s["ref"], s["flo"] = ref.contiguous(), flo.contiguous()
        s["params"] = _params(case)
        s["cdim"] = nrb.grid_dims(_dim(case), _pix(case), s["params"])
        s["cpp"] = torch.zeros(3 * int(np.prod(s["cdim"])), device="cuda")
        s["stream"] = torch.cuda.Stream()
    elif kind == "batch":
        s["params"] = _params(case)
        s["pairs"] = []
        for k in range(case["pairs"]):  # sizes around the case's, as a cohort's volumes differ
            c = dict(case, nx=case["nx"] - 5 * (k % 3), ny=case["ny"] + 4 * (k % 4), nz=case["nz"] + 7 * (k % 2))
            ref, flo = _pair(c, 100 * seed + k)
            s["pairs"].append((ref.cpu().numpy(), flo.cpu().numpy(), _pix(c)))
    elif kind == "f3d2":
        ref, flo = _pair(case, seed)
        s["ref"], s["flo"], s["params"] = ref.cpu().numpy(), flo.cpu().numpy(), _params(case)
        s["xyz"] = _rotation(case)
    return s


# ------------------------------------------------------------------------------------------------
# one pass
# ------------------------------------------------------------------------------------------------
def _objective_values(o):
    return {"nmi": o.nmi, "entropy": np.array(list(o.entropy)), "be": o.be, "objective": o.objective}


def run(s):
    case = s["case"]
    kind = case["kind"]
    stream = torch.cuda.current_stream()
    if kind == "objective":
        return _objective_values(nrb.f3d_objective(s["ws"], s["nmi"], s["ref"], s["flo"], s["cpp"], 1.0 - BE, BE,
                                                   mask=s["mask"], stream=stream))
    if kind == "gradient":
        nrb.f3d_gradient(s["ws"], s["nmi"], s["ref"], s["flo"], s["cpp"], s["vgrad"], s["node"], 1.0 - BE, BE,
                         mask=s["mask"], stream=stream)
        return {"vgrad": s["vgrad"], "node": s["node"]}
    if kind == "steps":
        g, mask, nmi, ws = s["g"], s["mask"], s["nmi"], s["ws"]
        n, nc = g.ref_nvox, g.cpp_nvox
        nrb.get_deformation_field(g, s["cpp"], s["def"], mask=mask, stream=stream)
        nrb.resample_image(g, s["flo"], s["def"], s["warped"], mask=mask, stream=stream)
        value = nrb.nmi_value(nmi, g, s["ref"], s["warped"], mask=mask, stream=stream)
        be = nrb.approx_bending_energy(ws, s["cpp"], stream=stream)
        nrb.get_image_gradient(g, s["flo"], s["def"], s["wgrad"], mask=mask, stream=stream)
        s["vgrad"].zero_()
        nrb.nmi_voxel_gradient(nmi, g, s["ref"], s["warped"], s["wgrad"], s["vgrad"], mask=mask, stream=stream)
        nrb.convolve_voxel_based_gradient(ws, s["vgrad"], s["node"], 1.0 - BE, stream=stream)
        nrb.approx_bending_energy_gradient(ws, s["cpp"], s["node"], BE, stream=stream)
        length = nrb.get_maximal_length(s["node"], nc, stream=stream)
        nrb.normalise_gradient(s["node"], nc, length, stream=stream)
        s["g1"].copy_(s["g1_0"])
        s["g2"].copy_(s["g2_0"])
        nrb.conjugate_gradient(ws, s["node"], s["g1"], s["g2"], 3 * nc, False, stream=stream)
        nrb.update_control_point_position(s["cur"], s["cpp"], s["node"], -0.5, 3 * nc, stream=stream)
        return {"nmi": value, "be": be, "def": s["def"], "warped": s["warped"], "wgrad": s["wgrad"],
                "vgrad": s["vgrad"], "direction": s["node"], "length": float(np.float32(length)), "cur": s["cur"]}
    if kind == "warp":
        nrb.f3d_warped_image(s["g"], s["flo"], s["cpp"], s["warped"], order=case["order"], padding=0.0, stream=stream)
        return s["warped"]
    if kind == "velocity":
        steps = nrb.get_def_field_from_velocity_grid(s["g"], s["vel"], 6, s["def"], update=True, stream=stream)
        return {"steps": steps, "def": s["def"]}
    if kind == "pyramid":
        nrb.image_pyramid(s["img"], _dim(case), _pix(case), s["xyz"], case["levels"], s["out"], stream=stream)
        s["finest"].copy_(s["img"].view(-1))
        nrb.intensity_rescale(s["finest"], s["finest"].numel(), 2.0, case["bins"] + 1.0, stream=stream)
        return {"levels": s["out"], "rescaled": s["finest"]}
    if kind == "register":
        s["stream"].wait_stream(stream)
        nrb.register_device(s["ref"], s["flo"], _dim(case), _pix(case), s["params"], s["cpp"], s["cpp"].numel(),
                            stream=s["stream"])
        return s["cpp"]
    if kind == "batch":
        return [cpp for cpp, _ in nrb.register_batch(s["pairs"], s["params"], concurrency=16)]
    fw, bw, _, steps, wf, wb, _ = nrb.f3d2_register_images(s["ref"], _pix(case), s["xyz"], s["flo"], _pix(case),
                                                           s["xyz"], s["params"])
    return {"forward": fw, "backward": bw, "steps": steps, "warped": wf, "warped_back": wb}


# ------------------------------------------------------------------------------------------------
# what a pass cannot do without
# ------------------------------------------------------------------------------------------------
def _evaluations(case):
    """Objective and gradient evaluations of a registration: the iteration budget counts both."""
    total, n = [], case["nx"] * case["ny"] * case["nz"]
    for level in range(case["levels"]):
        total.append((case["iterations"] * 2 ** level, n / 8.0 ** level))
    return total


def work(case):
    kind, n = case["kind"], float(case["nx"] * case["ny"] * case["nz"])
    extra = 4.0 * n if case.get("mask") else 0.0
    if kind == "pyramid":
        down = n * (1.0 / 7.0)
        return {"bytes": 4.0 * (n + n + down) + 8.0 * n, "flops": 20.0 * n}
    nodes = float(np.prod([math.ceil(case[k] * p / case["spacing"]) + 3 for k, p in zip(("nx", "ny", "nz"), _pix(case))]))
    # per voxel: the separable spline position (24), the trilinear sample (30), the bin (4)
    if kind == "objective":
        return {"bytes": 8.0 * n + 12.0 * nodes + extra, "flops": 60.0 * n}
    if kind == "gradient":  # and the spatial gradient, the Parzen window, the node convolution
        return {"bytes": 8.0 * n + 12.0 * n + 24.0 * nodes + extra, "flops": 220.0 * n}
    if kind == "steps":  # every intermediate image is an output: field, warp, gradients
        return {"bytes": (8.0 + 12.0 + 4.0 + 12.0 + 12.0) * n + 60.0 * nodes + extra, "flops": 220.0 * n}
    if kind == "warp":
        return {"bytes": 8.0 * n + 12.0 * nodes, "flops": (24.0 + (170.0 if case["order"] == 3 else 30.0)) * n}
    if kind == "velocity":
        return {"bytes": 12.0 * n + 12.0 * nodes, "flops": (400.0 + 6 * 60.0) * n}
    if kind in ("register", "batch"):
        pairs = case.get("pairs", 1)
        return {"bytes": pairs * sum(8.0 * m for _, m in _evaluations(case)), "flops":
                pairs * sum(0.3 * it * 60.0 * m for it, m in _evaluations(case))}
    return {"bytes": 2 * sum(8.0 * m for _, m in _evaluations(case)), "flops":
            2 * sum(0.3 * it * 760.0 * m for it, m in _evaluations(case))}


# ------------------------------------------------------------------------------------------------
# the same values in 64 bits
# ------------------------------------------------------------------------------------------------
def _spline(t):
    return torch.stack([(1 - t) ** 3 / 6, (3 * t ** 3 - 6 * t ** 2 + 4) / 6, (-3 * t ** 3 + 3 * t ** 2 + 3 * t + 1) / 6,
                        t ** 3 / 6], -1)


def _dense(n, ratio, nodes):
    """[n, nodes] cubic B-spline weights of voxels 0..n-1, `ratio` voxels per node."""
    v = torch.arange(n, device="cuda", dtype=torch.float64)
    pre = torch.floor(v / ratio)
    w = torch.zeros(n, nodes + 4, device="cuda", dtype=torch.float64)
    w.scatter_(1, pre.long()[:, None] + torch.arange(4, device="cuda"), _spline(v / ratio - pre))
    return w[:, :nodes]


def _mats(g):
    as64 = lambda a: torch.tensor(list(a), dtype=torch.float64, device="cuda").view(4, 4)  # noqa: E731
    return as64(g.ref_xyz), as64(g.flo_ijk), as64(g.cpp_xyz), as64(g.ref_ijk)


def _field(g, cpp):
    ratio = [float(np.float32(g.cpp_pixdim[i]) / np.float32(g.ref_pixdim[i])) for i in range(3)]
    w = [_dense(g.ref_dim[i], ratio[i], g.cpp_dim[i]) for i in range(3)]
    out = []
    for c in range(3):
        t = torch.tensordot(cpp[c].double(), w[0], dims=([2], [1]))   # cz cy nx
        t = torch.tensordot(w[1], t, dims=([1], [1]))                 # ny cz nx
        out.append(torch.tensordot(w[2], t, dims=([1], [1])))         # nz ny nx
    return out


def _to_voxel(m, p):
    return [m[k, 0] * p[0] + m[k, 1] * p[1] + m[k, 2] * p[2] + m[k, 3] for k in range(3)]


def _tap(img, x, y, z, pad):
    nz, ny, nx = img.shape
    ok = (x >= 0) & (x < nx) & (y >= 0) & (y < ny) & (z >= 0) & (z < nz)
    i = (z.clamp(0, nz - 1) * ny + y.clamp(0, ny - 1)) * nx + x.clamp(0, nx - 1)
    return torch.where(ok, img.view(-1)[i], pad)


def _linear(img, vox, pad, want_gradient):
    fl = [torch.floor(v) for v in vox]
    t = [v - f for v, f in zip(vox, fl)]
    base = [f.clamp(-1e6, 1e6).long() for f in fl]
    lerp = lambda a, b, k: a + t[k] * (b - a)  # noqa: E731  (exact where both ends agree)
    v = [[[_tap(img, base[0] + a, base[1] + b, base[2] + c, pad) for a in (0, 1)] for b in (0, 1)] for c in (0, 1)]
    row = [[lerp(v[c][b][0], v[c][b][1], 0) for b in (0, 1)] for c in (0, 1)]
    plane = [lerp(row[c][0], row[c][1], 1) for c in (0, 1)]
    val = lerp(plane[0], plane[1], 2)
    if not want_gradient:
        return val, None
    gx = [lerp(v[c][0][1] - v[c][0][0], v[c][1][1] - v[c][1][0], 1) for c in (0, 1)]
    grad = [lerp(gx[0], gx[1], 2), lerp(row[0][1] - row[0][0], row[1][1] - row[1][0], 2), plane[1] - plane[0]]
    return val, [torch.nan_to_num(q, nan=0.0) for q in grad]


def _warp_slabs(img, field, g, want_gradient, pad):
    """Trilinear warp (and spatial gradient) slab by slab, to bound the temporaries."""
    _, fijk, _, _ = _mats(g)
    img = img.double()
    vals, grads = [], [[], [], []]
    nz, ny, nx = field[0].shape
    step = max(1, int(12e6 // (ny * nx)))
    for z in range(0, nz, step):
        v, d = _linear(img, _to_voxel(fijk, [f[z:z + step] for f in field]), pad, want_gradient)
        vals.append(v)
        if want_gradient:
            for k in range(3):
                grads[k].append(d[k])
    return torch.cat(vals), [torch.cat(q) for q in grads] if want_gradient else None


def _tables(ref, warped, active, bins):
    """Smoothed joint probabilities, entropies and log tables of the approximate Parzen window."""
    ok = active & ~torch.isnan(warped) & (warped >= 0) & (warped < bins) & (ref >= 0) & (ref < bins)
    idx = ref[ok].long() + warped[ok].long() * bins
    h = torch.bincount(idx, minlength=bins * bins).double().view(bins, bins)  # [floating, reference]
    k0, k1 = 1.0 / 6.0, float(np.float32(2.0) / np.float32(3.0))
    for axis in (1, 0):
        p = torch.nn.functional.pad(h, (1, 1) if axis == 1 else (0, 0, 1, 1))
        a, b, c = (p[:, :-2], p[:, 1:-1], p[:, 2:]) if axis == 1 else (p[:-2], p[1:-1], p[2:])
        h = k0 * a + k1 * b + k0 * c
    total = h.sum()
    p = h / total
    log = lambda q: torch.where(q > 0, torch.log(q.clamp_min(1e-300)), torch.zeros_like(q))  # noqa: E731
    pr, pw = p.sum(0), p.sum(1)
    ent = [float(-(q * log(q)).sum()) for q in (pr, pw, p)]
    return (ent[0] + ent[1]) / ent[2], ent + [float(total)], log(p), log(pr), log(pw)


def _parzen(x):
    a = x.abs()
    two_thirds = float(np.float32(2.0) / np.float32(3.0))
    return torch.where(a < 1, two_thirds + (0.5 * a - 1) * a * a, torch.where(a < 2, (2 - a) ** 3 / 6, torch.zeros_like(a)))


def _parzen_slope(x):
    a = x.abs()
    return torch.where(a < 1, (1.5 * a - 2) * x, torch.where(a < 2, -0.5 * (a - 2) ** 2 * torch.sign(x), torch.zeros_like(a)))


def _voxel_gradient(ref, warped, grad, active, bins, tables, weight):
    nmi, ent, lj, lr, lw = tables
    out = [torch.zeros_like(grad[0]) for _ in range(3)]
    sel = (active & ~torch.isnan(warped)).view(-1).nonzero().view(-1)
    for part in sel.split(8_000_000):
        rv, wv = ref.view(-1)[part].double(), warped.view(-1)[part]
        r0, w0 = torch.trunc(rv - 1).long(), torch.trunc(wv - 1).long()
        s = 0.0
        for a in range(4):
            r = r0 + a
            br = _parzen(rv - r) * ((r >= 0) & (r < bins))
            r = r.clamp(0, bins - 1)
            for b in range(4):
                w = w0 + b
                dw = _parzen_slope(wv - w) * ((w >= 0) & (w < bins))
                w = w.clamp(0, bins - 1)
                s = s + br * dw * (lr[r] + lw[w] - nmi * lj[w, r])
        for k in range(3):
            out[k].view(-1)[part] = weight / (ent[2] * ent[3]) * grad[k].view(-1)[part] * s
    return out


def _sampling(g, axis):
    """[nodes, voxels]: the normalised cubic convolution along an axis, sampled at the nodes."""
    _, _, cxyz, rijk = _mats(g)
    n, nodes = g.ref_dim[axis], g.cpp_dim[axis]
    width = float(np.float32(g.cpp_pixdim[axis]) / np.float32(g.ref_pixdim[axis]))
    radius = int(np.float32(width) * 2)
    i = torch.arange(n, device="cuda", dtype=torch.float64)
    rel = (i[:, None] - i[None, :]).abs() / width
    k = torch.where(rel < 1, 2.0 / 3.0 - rel ** 2 + 0.5 * rel ** 3, torch.where(rel < 2, (2 - rel) ** 3 / 6, torch.zeros_like(rel)))
    k = k * ((i[:, None] - i[None, :]).abs() <= radius)
    k = k / k.sum(1, keepdim=True)
    m = (rijk @ cxyz)
    at = (m[axis, axis] * torch.arange(nodes, device="cuda", dtype=torch.float64) + m[axis, 3]).float().double()
    pre = torch.floor(at)
    out = torch.zeros(nodes, n, device="cuda", dtype=torch.float64)
    for c in (0, 1):
        w = (at - pre) if c else 1 - (at - pre)
        p = pre.long() + c
        ok = (p >= 0) & (p < n)
        out += (w * ok)[:, None] * k[p.clamp(0, n - 1)]
    return out


def _nodes(g, vgrad, weight):
    _, fijk, _, _ = _mats(g)
    ax = [_sampling(g, i) for i in range(3)]
    scale = weight * math.prod(float(g.cpp_pixdim[i]) / float(g.ref_pixdim[i]) for i in range(3))
    got = []
    for c in range(3):
        t = torch.tensordot(vgrad[c], ax[0], dims=([2], [1]))
        t = torch.tensordot(ax[1], t, dims=([1], [1]))
        got.append(torch.tensordot(ax[2], t, dims=([1], [1])))
    return torch.stack([scale * sum(fijk[r, d] * got[r] for r in range(3)) for d in range(3)])


def _stencils():
    """[6, 3, 3, 3] second-derivative stencils (z, y, x), rounded to six decimals."""
    b, d, s = np.array([1 / 6, 2 / 3, 1 / 6]), np.array([-0.5, 0.0, 0.5]), np.array([1.0, -2.0, 1.0])
    triples = [(b, b, s), (b, s, b), (s, b, b), (b, d, d), (d, d, b), (d, b, d)]
    return torch.tensor(np.stack([np.round(np.einsum("i,j,k->ijk", *t), 6) for t in triples]), device="cuda")


def _conv3(v, k):
    return torch.nn.functional.conv3d(v[:, None], k[:, None])


def _bending(g, cpp):
    """(energy, gradient of the energy times the node count) of the control-point grid."""
    v = cpp.view(3, g.cpp_dim[2], g.cpp_dim[1], g.cpp_dim[0]).double()
    m = _mats(g)[2]
    z, y, x = _axes(v.shape[1:])
    ident = torch.stack([(m[k, 0] * x + m[k, 1] * y + m[k, 2] * z + m[k, 3]).expand(v.shape[1:]) for k in range(3)])
    k = _stencils()
    twice = torch.tensor([1.0, 1, 1, 2, 2, 2], device="cuda", dtype=torch.float64).view(1, 6, 1, 1, 1)
    energy = float((twice * _conv3(v - ident, k) ** 2).sum() / (3.0 * g.cpp_nvox))
    d = _conv3(torch.nn.functional.pad(v - ident, (1, 1) * 3), k) * twice
    grad = torch.nn.functional.conv3d(torch.nn.functional.pad(d, (1, 1) * 3), k[None])[:, 0]
    return energy, grad


def _evaluate(case, s, want_gradient):
    bins = case["bins"] + MARGIN_BINS
    field = _field(s["g"], s["cpp"])
    warped, grad = _warp_slabs(s["flo"], field, s["g"], want_gradient, float("nan"))
    active = torch.ones_like(s["ref"], dtype=torch.bool) if s["mask"] is None else s["mask"] > -1
    return field, warped, grad, active, bins, _tables(s["ref"], warped, active, bins)


def _exact_velocity(case, s):
    g = s["g"]
    rxyz = _mats(g)[0]
    rijk = torch.linalg.inv(rxyz)
    cxyz = _mats(g)[2]
    cijk = torch.linalg.inv(cxyz)
    nz, ny, nx = g.ref_dim[2], g.ref_dim[1], g.ref_dim[0]
    z, y, x = [a.double() for a in _axes((nz, ny, nx))]
    ident = [(rxyz[k, 0] * x + rxyz[k, 1] * y + rxyz[k, 2] * z + rxyz[k, 3]).expand(nz, ny, nx) for k in range(3)]
    vox = _to_voxel(cijk, ident)
    pre = [torch.floor(v) for v in vox]
    w = [_spline(v - p) for v, p in zip(vox, pre)]
    pos = [0.0, 0.0, 0.0]
    vel = s["vel"].double()

    def slided(f, m, ix, iy, iz):
        d, h, n = f[0].shape
        cx, cy, cz = ix.clamp(0, n - 1), iy.clamp(0, h - 1), iz.clamp(0, d - 1)
        i = (cz * h + cy) * n + cx
        off = [(ix - cx).double(), (iy - cy).double(), (iz - cz).double()]
        return [f[k].reshape(-1)[i] + m[k, 0] * off[0] + m[k, 1] * off[1] + m[k, 2] * off[2] for k in range(3)]

    for c in range(4):
        for b in range(4):
            for a in range(4):
                v = slided(vel, cxyz, pre[0].long() - 1 + a, pre[1].long() - 1 + b, pre[2].long() - 1 + c)
                ww = w[0][..., a] * w[1][..., b] * w[2][..., c]
                pos = [p + ww * q for p, q in zip(pos, v)]
    disp = [p - i for p, i in zip(pos, ident)]
    top = max(float(q.abs().max()) for q in disp)
    steps = 6
    while top / 2 ** steps >= 0.28:
        steps += 1
    field = [q / 2 ** steps + i for q, i in zip(disp, ident)]
    for _ in range(steps):
        v = _to_voxel(rijk, field)
        p = [torch.floor(q) for q in v]
        t = [q - r for q, r in zip(v, p)]
        out = [0.0, 0.0, 0.0]
        for c in (0, 1):
            for b in (0, 1):
                for a in (0, 1):
                    q = slided(field, rxyz, p[0].long() + a, p[1].long() + b, p[2].long() + c)
                    ww = (t[0] if a else 1 - t[0]) * (t[1] if b else 1 - t[1]) * (t[2] if c else 1 - t[2])
                    out = [o + ww * e for o, e in zip(out, q)]
        field = out
    return {"steps": steps, "def": torch.stack(field).view(-1)}


def _exact_warp(case, s):
    g = s["g"]
    fijk = _mats(g)[1]
    vox = _to_voxel(fijk, _field(g, s["cpp"]))
    img = s["flo"].double()
    fl = [torch.floor(v) for v in vox]
    t = [v - f for v, f in zip(vox, fl)]
    base = [f.long() for f in fl]
    if case["order"] == 0:
        w = [torch.stack([(q < 0.5).double(), (q >= 0.5).double()], -1) for q in t]
    elif case["order"] == 1:
        w = [torch.stack([1 - q, q], -1) for q in t]
    else:
        w = [torch.stack([q * ((2 - q) * q - 1), q * q * (3 * q - 5) + 2, q * ((4 - 3 * q) * q + 1), (q - 1) * q * q], -1) / 2
             for q in t]
    taps, first = w[0].shape[-1], -1 if case["order"] == 3 else 0
    out = 0.0
    for c in range(taps):
        for b in range(taps):
            for a in range(taps):
                v = _tap(img, base[0] + first + a, base[1] + first + b, base[2] + first + c, 0.0)
                out = out + v * w[0][..., a] * w[1][..., b] * w[2][..., c]
    return out.view(-1)


def _exact_pyramid(case, s):
    sigma = 0.7355
    radius = int(sigma * 3.0)
    k = torch.tensor([math.exp(-i * i / (2 * sigma * sigma)) / (sigma * 2.506628274631) for i in range(-radius, radius + 1)],
                     device="cuda", dtype=torch.float64).float().double()
    level, levels = s["img"].double(), [s["img"].double()]
    for _ in range(case["levels"] - 1):
        for axis in range(3):
            # the value over the weights inside the volume, along one axis at a time
            n = level.shape[axis]
            i = torch.arange(n, device="cuda")
            off = i[None, :] - i[:, None]
            m = torch.where(off.abs() <= radius, k[(off + radius).clamp(0, 2 * radius)], 0.0)
            m = m / m.sum(1, keepdim=True)
            if n // 2 >= 32:
                m = m[::2]
            level = torch.movedim(torch.tensordot(m, level, dims=([1], [axis])), 0, axis)
        levels.insert(0, level)
    d = s["img"].double().view(-1)
    lo, hi = d.min(), d.max()
    return {"levels": torch.cat([q.reshape(-1) for q in levels]),
            "rescaled": (d - lo) / (hi - lo) * (case["bins"] - 1.0) + 2.0}


def exact(case, seed):
    kind = case["kind"]
    if kind in ("register", "batch", "f3d2"):
        return None  # an optimiser's path: no value of its own in another precision
    s = prepare(case, seed)
    if kind == "warp":
        return _exact_warp(case, s)
    if kind == "velocity":
        return _exact_velocity(case, s)
    if kind == "pyramid":
        return _exact_pyramid(case, s)
    g = s["g"]
    field, warped, grad, active, bins, tables = _evaluate(case, s, kind != "objective")
    if kind == "objective":
        be = _bending(g, s["cpp"])[0]
        return {"nmi": tables[0], "entropy": torch.tensor(tables[1], dtype=torch.float64), "be": be,
                "objective": (1.0 - BE) * tables[0] - BE * be}
    keep_field = field if kind == "steps" else None
    del field
    vg = _voxel_gradient(s["ref"], warped, grad, active, bins, tables, 1.0)
    be, bg = _bending(g, s["cpp"])
    node = _nodes(g, vg, 1.0 - BE) + BE / g.cpp_nvox * bg
    if kind == "gradient":
        return {"vgrad": torch.stack(vg).view(-1), "node": node.view(-1)}
    zero = torch.zeros((), device="cuda", dtype=torch.float64)
    flat = lambda q: torch.stack([torch.where(active, p, zero) for p in q]).view(-1)  # noqa: E731
    # the conjugate direction turns on two dot products of float gradients, and with it the
    # updated grid: no value of their own in another precision
    return {"nmi": tables[0], "be": be, "def": flat(keep_field), "warped": torch.where(active, warped, zero).view(-1),
            "wgrad": flat(grad), "vgrad": flat(vg), "direction": None, "length": None, "cur": None}
