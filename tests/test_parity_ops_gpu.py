"""Parity of every C-ABI operation with the CPU oracle (oracle/nrb_oracle.c) on seeded inputs.

Tolerances (stated per test): deformation field within 1e-4 voxel; resampled intensities and
spatial gradients within 1e-4 absolute on [2, 65]-scaled images with identical NaN patterns;
integer joint histograms exact; NMI, entropies and log tables within 1e-10 relative; voxel
and node gradients within 1e-5 of the largest magnitude; bending energy within 1e-6 relative.
"""
import math

import numpy as np
import pytest

import niftyreg_b200 as nrb
import oracle
from tests.helpers import ensure_built, identity_grid, make_case

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

CASES = {
    "iso5": dict(),
    "spacing2": dict(shape=(16, 17, 19), spacing_vox=(2.0, 2.0, 2.0), seed=1),
    "aniso": dict(shape=(18, 30, 26), pixdim=(0.8, 0.8, 1.5), spacing_vox=(12.5, 12.5, 20.0 / 3.0), seed=2),
    "flo_geom": dict(shape=(20, 22, 24), flo_shape=(18, 22, 26), flo_pixdim=(1.2, 1.1, 0.9), seed=3, disp=0.8),
    "nan_ref": dict(seed=4, nan_frac=0.02),
    "bins132": dict(seed=5, bins=132),
}


@pytest.fixture(scope="module")
def O():
    ensure_built()
    return oracle.Restated()


def dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def host(t):
    torch.cuda.synchronize()
    return t.cpu().numpy()


@pytest.fixture(params=list(CASES), scope="module")
def case(request):
    return make_case(**CASES[request.param])


def oracle_pipeline(O, c):
    dfield = O.deformation_field(c.cpp, c.cdim, c.cpix, c.rdim, c.rpix)
    warped = O.resample(c.flo, c.fdim, c.flo_ijk, dfield, c.rdim)
    return dfield, warped


def test_deformation_field(O, case):
    c = case
    g = c.geometry()
    d = torch.empty(3 * c.nvox, dtype=torch.float32, device="cuda")
    nrb.get_deformation_field(g, dev(c.cpp), d)
    ref = O.deformation_field(c.cpp, c.cdim, c.cpix, c.rdim, c.rpix)
    diff = np.abs(host(d) - ref).reshape(3, -1)
    vox = diff / np.asarray(c.rpix, np.float32)[:, None]
    assert vox.max() <= 1e-4, f"max field error {vox.max():.3g} voxel"


def test_deformation_field_mask(O):
    c = make_case(seed=7)
    rng = np.random.default_rng(7)
    mask = np.where(rng.random(c.nvox) < 0.3, -1, 0).astype(np.int32)
    g = c.geometry()
    d = torch.empty(3 * c.nvox, dtype=torch.float32, device="cuda")
    nrb.get_deformation_field(g, dev(c.cpp), d, mask=dev(mask))
    ref = O.deformation_field(c.cpp, c.cdim, c.cpix, c.rdim, c.rpix, mask=mask)
    out = host(d).reshape(3, -1)
    assert np.all(out[:, mask < 0] == 0)
    assert np.abs(out - ref.reshape(3, -1)).max() <= 1e-4


def test_resample_and_gradient(O, case):
    c = case
    g = c.geometry()
    dfield, warped_ref = oracle_pipeline(O, c)
    w = torch.empty(c.nvox, dtype=torch.float32, device="cuda")
    nrb.resample_image(g, dev(c.flo), dev(dfield), w)
    wg = host(w)
    assert np.array_equal(np.isnan(wg), np.isnan(warped_ref)), "NaN padding pattern differs"
    ok = np.isfinite(warped_ref)
    assert np.abs(wg[ok] - warped_ref[ok]).max() <= 1e-4
    gr = torch.empty(3 * c.nvox, dtype=torch.float32, device="cuda")
    nrb.get_image_gradient(g, dev(c.flo), dev(dfield), gr)
    gref = O.image_gradient(c.flo, c.fdim, c.flo_ijk, dfield, c.rdim)
    assert np.abs(host(gr) - gref).max() <= 1e-4


def test_resample_padding_and_mask(O):
    c = make_case(seed=8, disp=4.0)
    rng = np.random.default_rng(8)
    mask = np.where(rng.random(c.nvox) < 0.25, -1, 0).astype(np.int32)
    g = c.geometry()
    dfield, _ = oracle_pipeline(O, c)
    init = np.full(c.nvox, -7.0, np.float32)
    for pad in (0.0, math.nan):
        w = dev(init.copy())
        nrb.resample_image(g, dev(c.flo), dev(dfield), w, padding=pad, mask=dev(mask))
        ref = O.resample(c.flo, c.fdim, c.flo_ijk, dfield, c.rdim, mask=mask, pad=pad, warped_init=init)
        out = host(w)
        assert np.all(out[mask < 0] == -7.0), "masked voxels must be left untouched"
        assert np.array_equal(np.isnan(out), np.isnan(ref))
        ok = np.isfinite(ref)
        assert np.abs(out[ok] - ref[ok]).max() <= 1e-4


def test_intensity_rescale(O):
    rng = np.random.default_rng(11)
    img = (rng.normal(100, 40, 5000)).astype(np.float32)
    img[::97] = np.nan
    t = dev(img)
    nrb.intensity_rescale(t, img.size, 2.0, 65.0)
    ref = O.intensity_rescale(img, 2.0, 65.0)
    out = host(t)
    assert np.array_equal(np.isnan(out), np.isnan(ref))
    ok = np.isfinite(ref)
    assert np.array_equal(out[ok], ref[ok]), "double-precision rescale must be bit-exact"


def test_nmi_value_and_tables(O, case):
    c = case
    g = c.geometry()
    _, warped = oracle_pipeline(O, c)
    nmi = nrb.Nmi(c.bins, c.bins)
    v = nrb.nmi_value(nmi, g, dev(c.ref), dev(warped))
    pro, log, ent = nmi.tables()
    v_ref, pro_ref, log_ref, ent_ref = O.nmi_value(c.ref, warped, c.bins, c.bins)
    assert abs(v - v_ref) <= 1e-10 * abs(v_ref)
    assert np.allclose(ent, ent_ref, rtol=1e-10, atol=0)
    assert np.allclose(pro, pro_ref, rtol=1e-10, atol=1e-18)
    assert np.allclose(log, log_ref, rtol=1e-10, atol=1e-12)


def test_nmi_voxel_gradient(O, case):
    _check_nmi_voxel_gradient(O, case)


def test_nmi_voxel_gradient_large_table(O):
    """180 internal bins: the FP32 copy of the log table (131 KB) does not fit in shared memory,
    so the FP64 window on the global table runs; the same bar."""
    _check_nmi_voxel_gradient(O, make_case(seed=6, bins=180))


def _check_nmi_voxel_gradient(O, c):
    g = c.geometry()
    dfield, warped = oracle_pipeline(O, c)
    wgrad = O.image_gradient(c.flo, c.fdim, c.flo_ijk, dfield, c.rdim)
    nmi = nrb.Nmi(c.bins, c.bins)
    nrb.nmi_value(nmi, g, dev(c.ref), dev(warped))
    vg = torch.zeros(3 * c.nvox, dtype=torch.float32, device="cuda")
    nrb.nmi_voxel_gradient(nmi, g, dev(c.ref), dev(warped), dev(wgrad), vg, weight=0.75)
    _, _, log_ref, ent_ref = O.nmi_value(c.ref, warped, c.bins, c.bins)
    ref = O.nmi_voxel_gradient(c.ref, warped, wgrad, c.bins, c.bins, log_ref, ent_ref, 0.75)
    scale = np.abs(ref).max()
    assert scale > 0
    assert np.abs(host(vg) - ref).max() <= 1e-5 * scale


def test_kernel_convolution_cubic(O):
    rng = np.random.default_rng(12)
    dim, pix = (23, 19, 17), (1.0, 1.2, 0.9)
    img = rng.normal(0, 1, 3 * int(np.prod(dim))).astype(np.float32)
    img[rng.random(img.size) < 0.02] = np.nan
    for axis in range(3):
        t = dev(img)
        nrb.kernel_convolution_cubic(t, 3, dim, pix, 5.0, axis)
        ref = O.kernel_convolution_cubic(img, 3, dim, pix, 5.0, axis)
        out = host(t)
        assert np.array_equal(np.isnan(out), np.isnan(ref))
        ok = np.isfinite(ref)
        assert np.abs(out[ok] - ref[ok]).max() <= 1e-5 * np.abs(ref[ok]).max()


def test_convolve_to_nodes(O, case):
    c = case
    g = c.geometry()
    rng = np.random.default_rng(13)
    vgrad = rng.normal(0, 1e-3, 3 * c.nvox).astype(np.float32)
    ws = nrb.Workspace(g)
    node = torch.full((3 * c.ncp,), 123.0, dtype=torch.float32, device="cuda")
    nrb.convolve_voxel_based_gradient(ws, dev(vgrad), node, 0.995)
    _, ref = O.convolve_to_nodes(vgrad, c.rdim, c.rpix, c.ref_ijk, c.cdim, c.cpix, c.cxyz, c.flo_ijk, 0.995)
    scale = np.abs(ref).max()
    assert np.abs(host(node) - ref).max() <= 1e-5 * scale


@pytest.mark.parametrize("dim,spacing", [((33, 5, 3), 5.0), ((3, 34, 7), 2.5), ((2, 9, 65), 40.0), ((700, 3, 2), 5.0),
                                         ((3, 1100, 5), 5.0), ((5, 2, 1500), 5.0), ((7000, 2, 2), 5.0), ((2, 7000, 3), 5.0),
                                         ((700, 50, 51), 5.0), ((50, 700, 51), 5.0), ((41, 30, 1500), 5.0),
                                         ((1500, 41, 30), 5.0)])
def test_kernel_convolution_cubic_line_lengths(O, dim, spacing):
    """Lines held 32, 16 and 8 at a time with remainders, windows longer than the line, lines too
    long for a block or too few for the device (the separate passes); NaN voxels. The bar of the op above; the allocation-free entry point gives the
    same floats."""
    import ctypes
    rng = np.random.default_rng(sum(dim))
    pix = (1.0, 1.0, 1.0)
    img = rng.normal(0, 1, 2 * int(np.prod(dim))).astype(np.float32)
    img[rng.random(img.size) < 0.02] = np.nan
    for axis in range(3):
        t, u = dev(img), dev(img)
        nrb.kernel_convolution_cubic(t, 2, dim, pix, spacing, axis)
        nrb.check(nrb.lib().nrb_kernel_convolution_cubic_static(
            ctypes.c_void_p(u.data_ptr()), 2, nrb._I3(*dim), nrb._F3(*pix), ctypes.c_float(spacing), axis, None))
        ref = O.kernel_convolution_cubic(img, 2, dim, pix, spacing, axis)
        out = host(t)
        assert np.array_equal(out, host(u), equal_nan=True)
        assert np.array_equal(np.isnan(out), np.isnan(ref))
        ok = np.isfinite(ref)
        assert np.abs(out[ok] - ref[ok]).max() <= 1e-5 * np.abs(ref[ok]).max()


@pytest.mark.parametrize("bins", [68, 212])
def test_nmi_voxel_gradient_of_intensities_far_outside_the_bins(O, bins):
    """Infinite and huge intensities on either side lie in no Parzen window: their voxels keep the
    gradient they had, and the others' floats are those of the same images with NaN in their place
    (which is skipped). The FP32 window (68 bins) and the FP64 one (a table of 212 is too large for
    shared memory), and the fused gradient of such a reference."""
    rng = np.random.default_rng(bins)
    c = make_case(shape=(12, 14, 16), seed=21, bins=bins)
    g = c.geometry()
    far = np.float32([np.inf, -np.inf, 3e9, -3e9, 1e30, 2147483520.0, 2147483648.0, -2147483648.0, 5e3, -40.0])
    at = rng.permutation(c.nvox)[:4 * far.size].reshape(2, -1)
    ref, war = c.ref.copy(), rng.uniform(2, bins - 3, c.nvox).astype(np.float32)
    ref[np.isnan(ref)] = 3.0
    wgrad, init = (rng.normal(0, 1, 3 * c.nvox).astype(np.float32) for _ in range(2))

    def gradient(r, w):
        nmi = nrb.Nmi(bins, bins)
        v = dev(init)
        nrb.nmi_value(nmi, g, dev(r), dev(w))
        nrb.nmi_voxel_gradient(nmi, g, dev(r), dev(w), dev(wgrad), v)
        return host(v).reshape(3, -1)

    def fused(r):
        nmi, ws = nrb.Nmi(bins, bins), nrb.Workspace(g)
        v, n = (torch.empty(3 * k, dtype=torch.float32, device="cuda") for k in (c.nvox, c.ncp))
        nrb.f3d_gradient(ws, nmi, dev(r), dev(c.flo), dev(c.cpp), v, n, 1.0, 0.0)
        return host(v).reshape(3, -1)

    out = []
    for values in (np.tile(far, 2), np.full(2 * far.size, np.nan, np.float32)):
        r, w = ref.copy(), war.copy()
        r[at[0]], w[at[1]] = values, values
        out.append((gradient(r, w), fused(r)))
    for a, b in zip(*out):
        assert np.array_equal(a, b)
    assert np.array_equal(out[0][0][:, at.ravel()], init.reshape(3, -1)[:, at.ravel()])
    assert not out[0][1][:, at[0]].any()


def test_bending_energy_gradient_with_another_grids_workspace(O):
    """The gradient's scratch comes from any workspace: grids of other dims (longer and thinner, larger,
    smaller) through one made for 9x10x11 nodes, and that grid again after each. The oracle's bar
    of the op below, and bit for bit what a workspace of the grid's own gives."""
    import ctypes
    pix, rng = (1.0, 1.0, 1.0), np.random.default_rng(8)
    xyz = nrb.identity_header(pix)

    class Grid:
        def __init__(self, cdim):
            rdim = tuple(5 * (n - 3) for n in cdim)
            cxyz = nrb.identity_header((5.0,) * 3, (-5.0,) * 3)
            self.g = nrb.make_geometry(rdim, pix, xyz, rdim, pix, xyz, cdim, (5.0,) * 3, cxyz)
            self.n = 3 * int(np.prod(cdim))
            cpp = (identity_grid(cdim, cxyz) + rng.normal(0, 2, self.n)).astype(np.float32)
            self.cpp = dev(cpp)
            self.ws = nrb.Workspace(self.g)
            self.own = self.gradient(self.ws)
            want = O.be_gradient(cpp, cdim, cxyz, 0.05)
            assert np.abs(self.own - want).max() <= 1e-5 * np.abs(want).max()

        def gradient(self, ws):
            t = torch.zeros(self.n, dtype=torch.float32, device="cuda")
            nrb.check(nrb.lib().nrb_approx_bending_energy_gradient(ws.h, ctypes.byref(self.g), nrb._p(self.cpp),
                                                                   ctypes.c_float(0.05), nrb._p(t), None))
            return host(t)

    first = Grid((9, 10, 11))
    for cdim in ((40, 5, 4), (14, 13, 12), (4, 4, 4), (11, 10, 9)):
        other = Grid(cdim)
        assert np.array_equal(other.gradient(first.ws), other.own)
        assert np.array_equal(first.gradient(first.ws), first.own)


def test_threads_with_different_sizes_do_not_disturb_each_other():
    """Two host threads, each on its own stream, run the same kernels with different shared-memory
    sizes (line lengths, volume widths, bin counts) at once: every call succeeds and gives the floats
    that it gives alone."""
    import threading
    pix = (1.0, 1.0, 1.0)
    xyz = nrb.identity_header(pix)

    class Work:
        def __init__(self, line, width, bins, seed):
            rng = np.random.default_rng(seed)
            self.line = (40, line, 80)  # blocks enough for the whole-line pass
            self.img = dev(rng.normal(0, 1, int(np.prod(self.line))).astype(np.float32))
            dim = (width, width, 2)
            cdim, cpix, cxyz = nrb.control_grid_header(dim, pix, (5.0, 5.0, 5.0))
            self.g = nrb.make_geometry(dim, pix, xyz, dim, pix, xyz, cdim, cpix, cxyz)
            n = int(np.prod(dim))
            self.ws, self.nmi = nrb.Workspace(self.g), nrb.Nmi(bins, bins)
            self.vg = dev(rng.normal(0, 1e-3, 3 * n).astype(np.float32))
            self.node = torch.empty(3 * int(np.prod(cdim)), dtype=torch.float32, device="cuda")
            self.ref, self.war = (dev(rng.uniform(2, bins - 3, n).astype(np.float32)) for _ in range(2))
            self.stream = torch.cuda.Stream()
            torch.cuda.synchronize()
            self.want = self.run()

        def run(self):
            with torch.cuda.stream(self.stream):
                img, out = self.img.clone(), torch.zeros_like(self.vg)
                nrb.kernel_convolution_cubic(img, 1, self.line, pix, 5.0, 1, stream=self.stream)
                nrb.convolve_voxel_based_gradient(self.ws, self.vg, self.node, 0.995, stream=self.stream)
                v = nrb.nmi_value(self.nmi, self.g, self.ref, self.war, stream=self.stream)
                nrb.nmi_voxel_gradient(self.nmi, self.g, self.ref, self.war, self.vg, out, stream=self.stream)
                self.stream.synchronize()
                return [t.cpu().numpy() for t in (img, self.node, out)] + [v]

        def loop(self):
            try:
                for _ in range(200):
                    assert all(np.array_equal(a, b) for a, b in zip(self.run(), self.want))
            except BaseException as e:  # reported by the test's own thread
                self.error = e

    work = [Work(400, 256, 132, 1), Work(150, 240, 68, 2)]
    threads = [threading.Thread(target=w.loop) for w in work]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for w in work:
        if getattr(w, "error", None):
            raise w.error


@pytest.mark.parametrize("fdim", [(2, 2, 2), (1, 5, 4), (3, 2, 9), (40, 7, 5)])
@pytest.mark.parametrize("pad", [np.nan, 0.0, 3.5])
def test_trilinear_warp_at_the_volume_border(O, fdim, pad):
    """The warp and its gradient against the oracle for floating volumes down to one voxel per axis,
    positions on voxels, between them, in the last cell and far outside: NaN padding (which takes
    footprints moved inside the volume where every axis has two voxels) and finite padding. The NaN
    pattern is exact; values within 1e-5 of the largest magnitude (sums of eight float products)."""
    rng = np.random.default_rng(fdim[0])
    c = make_case(shape=(6, 7, 40), seed=39)
    pix = (1.0, 1.0, 1.0)
    g = nrb.make_geometry(c.rdim, c.rpix, c.rxyz, fdim, pix, nrb.identity_header(pix), c.cdim, c.cpix, c.cxyz)
    flo = rng.normal(0, 100, int(np.prod(fdim))).astype(np.float32)
    pos = np.stack([rng.uniform(-2, n + 1, c.nvox) for n in fdim]).astype(np.float32)
    pos[:, :64] = np.round(pos[:, :64])
    pos[:, 64:96] = -1.0e7
    for a, n in enumerate(fdim):
        pos[a, 96:800] = rng.uniform(0, max(n - 1, 0.001), 704)
    w = torch.empty(c.nvox, dtype=torch.float32, device="cuda")
    wg = torch.empty(3 * c.nvox, dtype=torch.float32, device="cuda")
    nrb.resample_image(g, dev(flo), dev(pos.ravel()), w, padding=pad)
    nrb.get_image_gradient(g, dev(flo), dev(pos.ravel()), wg, padding=pad)
    eye = np.eye(4, dtype=np.float32)
    near = np.abs(pos).max(0) < 1.0e6  # a fraction 1e7 voxels out is no fraction
    for out, ref in ((host(w), O.resample(flo, fdim, eye, pos.ravel(), c.rdim, pad=pad)),
                     (host(wg), O.image_gradient(flo, fdim, eye, pos.ravel(), c.rdim, pad=pad))):
        out, ref = out.reshape(-1, c.nvox)[:, near], ref.reshape(-1, c.nvox)[:, near]
        assert np.array_equal(np.isnan(out), np.isnan(ref))
        ok = ~np.isnan(ref)
        assert np.abs(out[ok] - ref[ok]).max(initial=0) <= 1e-5 * 500.0


def convolve_then_sample(O, v, dim, pix, cdim, cpix, weight):
    """The node gradient of an identity-oriented image whose grid starts one spacing before it: the
    oracle's convolution along each axis, then the trilinear sample at every node over the taps of
    non-zero weight inside the volume (a tap of zero weight is not read, so a NaN there does not
    count; the oracle's own node sampling multiplies it)."""
    nx, ny, nz = dim
    for axis in range(3):
        v = O.kernel_convolution_cubic(v, 3, dim, pix, cpix[axis], axis)
    vol = np.asarray(v, np.float64).reshape(3, nz, ny, nx)
    out = vol
    with np.errstate(invalid="ignore"):
        for axis, (n, nodes, step, d) in enumerate(zip(dim, cdim, cpix, pix)):
            step = float(np.float32(step))  # as the geometry holds it
            at = (np.arange(nodes) * (step / d) - step / d).astype(np.float32).astype(np.float64)
            pre = np.floor(at).astype(int)
            parts = []
            for p, w1 in zip(pre, at - pre):
                acc = np.zeros(np.delete(out.shape, 3 - axis))
                for q, w in ((p, 1.0 - w1), (p + 1, w1)):
                    if 0 <= q < n and w != 0.0:
                        acc = acc + w * np.take(out, q, axis=3 - axis)
                parts.append(acc)
            out = np.stack(parts, axis=3 - axis)
        # reorientation by the identity: an infinite component meets the other rows' zeros
        out = np.stack([sum(np.eye(3)[c, d] * out[c] for c in range(3)) for d in range(3)])
        return (out * weight * np.prod([c / p for c, p in zip(cpix, pix)])).ravel()


@pytest.mark.parametrize("shape,spacing", [((3, 11, 200), 5.0), ((2, 5, 401), 5.0), ((2, 3, 900), 7.3), ((3, 301, 222), 3.0),
                                           ((33, 6, 7), 2.5), ((9, 10, 12), 30.0), ((2, 3, 2040), 1020.0),
                                           ((100, 60, 61), 2.5), ((26, 301, 222), 3.0)])
def test_convolve_to_nodes_at_tile_edges(O, shape, spacing):
    """Rows staged 32, 16, 8 and 4 at a time with a remainder, a y pass by whole slices, by shares of
    their columns and by single outputs, outputs not a multiple of four, two samples per node (a spacing that is no whole number of voxels), windows
    longer than the lines; finite gradients, then NaN and infinite ones. The bar of the op above."""
    rng = np.random.default_rng(shape[2])
    nz, ny, nx = shape
    dim, pix = (nx, ny, nz), (1.0, 1.0, 1.0)
    xyz = nrb.identity_header(pix)
    cdim, cpix, cxyz = nrb.control_grid_header(dim, pix, (spacing,) * 3)
    g = nrb.make_geometry(dim, pix, xyz, dim, pix, xyz, cdim, cpix, cxyz)
    ws = nrb.Workspace(g)
    n, nc = nx * ny * nz, int(np.prod(cdim))
    vgrad = rng.normal(0, 1e-3, 3 * n).astype(np.float32)
    spoiled = vgrad.copy()
    spoiled[rng.integers(0, 3 * n, 5)] = np.nan
    spoiled[rng.integers(0, 3 * n, 2)] = np.inf
    for v in (vgrad, spoiled):
        node = torch.full((3 * nc,), 123.0, dtype=torch.float32, device="cuda")
        nrb.convolve_voxel_based_gradient(ws, dev(v), node, 0.995)
        ref = convolve_then_sample(O, v, dim, pix, cdim, cpix, 0.995)
        out = host(node)
        ok = np.isfinite(ref)
        assert np.array_equal(np.isfinite(out), ok)
        assert np.array_equal(np.isnan(out), np.isnan(ref))
        if ok.any():
            assert np.abs(out[ok] - ref[ok]).max() <= 1e-5 * np.abs(ref[ok]).max()


def nodes_in_float(v, shape, cdim, spacing, weight):
    """The node gradient of a 1 mm image whose nodes sit on every `spacing`-th voxel, in the float
    operations of the convolution: per axis and sampled voxel the taps in ascending order, each a
    fused multiply-add over the values that are not NaN, divided by the sum of their weights; a NaN
    voxel stays NaN. A node reads one voxel, times the weight. (The product of two floats is exact in
    long double, and its sum with a third far closer than a float.)"""
    t = np.abs(np.arange(-2 * spacing, 2 * spacing + 1) / float(spacing))
    taps = np.where(t < 1, 2.0 / 3.0 - t * t + 0.5 * t * t * t, -(t - 2.0) ** 3 / 6.0).astype(np.float32)
    out = v.reshape((3,) + shape)
    for axis in (3, 2, 1):
        line = np.moveaxis(out, axis, 0)
        n, res = line.shape[0], []
        for s in range(0, n, spacing):
            num, den = np.zeros(line.shape[1:], np.float32), np.zeros(line.shape[1:], np.float32)
            for k in range(max(0, s - 2 * spacing), min(n - 1, s + 2 * spacing) + 1):
                w, x = taps[k - s + 2 * spacing], line[k]
                ok = ~np.isnan(x)
                fma = (np.longdouble(w) * x.astype(np.longdouble) + num).astype(np.float32)
                num, den = np.where(ok, fma, num), np.where(ok, den + w, den)
            res.append(np.where(np.isnan(line[s]), np.float32(np.nan), num / den))
        out = np.moveaxis(np.stack(res), 0, axis)
    out = np.where(np.isnan(out).any(0), np.float32(np.nan), out)  # the reorientation mixes the components
    node = np.zeros((3,) + tuple(cdim[::-1]), np.float32)
    nz, ny, nx = out.shape[1:]
    node[:, 1:1 + nz, 1:1 + ny, 1:1 + nx] = out * np.float32(weight * spacing ** 3)
    return node


def test_convolve_to_nodes_nan_free_path_is_exact():
    """Outputs whose window holds no NaN take a check-free sum, the others the per-tap path (conv_at).
    Against one restatement in float, bit for bit, for a gradient without NaN (the check-free path
    alone) and with NaN voxels (both paths side by side), and nodes out of a NaN's reach keep their
    floats."""
    c = make_case(shape=(24, 24, 48), seed=31)
    g = c.geometry()
    rng = np.random.default_rng(31)
    vgrad = rng.normal(0, 1e-3, 3 * c.nvox).astype(np.float32)
    ws = nrb.Workspace(g)
    spoiled = vgrad.copy()
    spoiled[3 * 48] = np.nan  # component 0, z = 0, y = 3, x = 0
    scattered = vgrad.copy()
    scattered[rng.integers(0, 3 * c.nvox, 40)] = np.nan
    scattered[5 * 48:5 * 48 + 5] = np.nan
    cx, cy, cz = c.cdim
    got = []
    for v in (vgrad, spoiled, scattered):
        node = torch.empty(3 * c.ncp, dtype=torch.float32, device="cuda")
        nrb.convolve_voxel_based_gradient(ws, dev(v), node, 0.5)
        got.append(host(node).reshape(3, cz, cy, cx))
        want = nodes_in_float(v, (24, 24, 48), c.cdim, 5, 0.5)
        assert np.array_equal(got[-1], want, equal_nan=True)
    assert not np.array_equal(got[0][0, :, :, :3], got[1][0, :, :, :3])  # the NaN changed the nodes near it
    assert np.array_equal(got[0][..., 5:], got[1][..., 5:])


def test_bending_energy(O, case):
    c = case
    g = c.geometry()
    ws = nrb.Workspace(g)
    be = nrb.approx_bending_energy(ws, dev(c.cpp))
    be_ref = O.be_value(c.cpp, c.cdim)
    assert abs(be - be_ref) <= 1e-6 * abs(be_ref)
    grad0 = np.random.default_rng(14).normal(0, 1, 3 * c.ncp).astype(np.float32)
    gt = dev(grad0)
    nrb.approx_bending_energy_gradient(ws, dev(c.cpp), gt, 0.005)
    ref = O.be_gradient(c.cpp, c.cdim, c.cxyz, 0.005, grad_init=grad0)
    delta, delta_ref = host(gt) - grad0, ref - grad0
    assert np.abs(delta - delta_ref).max() <= 1e-5 * np.abs(delta_ref).max()


def test_bending_energy_identity_is_zero():
    # known answer of reg_test_be.cpp: identity and affine grids have zero bending energy
    c = make_case(seed=15, disp=0.0)
    g = c.geometry()
    ws = nrb.Workspace(g)
    assert abs(nrb.approx_bending_energy(ws, dev(c.cpp))) < 1e-9
    grad = torch.zeros(3 * c.ncp, dtype=torch.float32, device="cuda")
    nrb.approx_bending_energy_gradient(ws, dev(c.cpp), grad, 1.0)
    assert host(grad).max() == 0 and host(grad).min() == 0


def test_optimiser_ops(O):
    rng = np.random.default_rng(16)
    nnode = 3000
    grad = rng.normal(0, 2, 3 * nnode).astype(np.float32)
    ml = nrb.get_maximal_length(dev(grad), nnode)
    assert ml == O.max_length(grad, nnode)
    t = dev(grad)
    nrb.normalise_gradient(t, nnode, ml)
    assert np.array_equal(host(t), O.normalise_gradient(grad, nnode, ml))
    best = rng.normal(0, 50, 3 * nnode).astype(np.float32)
    cur = torch.empty_like(t)
    nrb.update_control_point_position(cur, dev(best), dev(grad), -0.37, 3 * nnode)
    assert np.array_equal(host(cur), O.update_control_points(best, grad, -0.37))


def test_conjugate_gradient(O):
    c = make_case(seed=17)
    ws = nrb.Workspace(c.geometry())
    rng = np.random.default_rng(17)
    n = 3 * c.ncp
    g0 = rng.normal(0, 1, n).astype(np.float32)
    g, a1, a2 = dev(g0), torch.empty(n, device="cuda"), torch.empty(n, device="cuda")
    nrb.conjugate_gradient(ws, g, a1, a2, n, True)
    rg, r1, r2 = O.cg_update(g0, np.zeros(n, np.float32), np.zeros(n, np.float32), True)
    assert np.array_equal(host(a1), r1) and np.array_equal(host(a2), r2)
    g1 = rng.normal(0, 1, n).astype(np.float32)
    g = dev(g1)
    nrb.conjugate_gradient(ws, g, a1, a2, n, False)
    rg, r1, r2 = O.cg_update(g1, r1, r2, False)
    # the dot products are reduced in a different (fixed) order: FP64 rounding only
    assert np.abs(host(g) - rg).max() <= 1e-6 * np.abs(rg).max()
    assert np.array_equal(host(a1), r1)
