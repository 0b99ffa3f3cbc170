"""Pyramid construction and control-point grid refinement (the registration's level set-up)
against the reference CPU library (oracle/_ref):

* nrb_image_pyramid vs reg_createImagePyramid<float> (reg-lib/cpu/_reg_tools.cpp:1705-1733, with
  reg_downsampleImage, :1343-1500): level dims and sform matrices equal (CPU, host-only
  headers); level data with the same NaN pattern and every value within 1e-6 of the level's
  largest magnitude (GPU; the Gaussian smoothing sums in double in both, and the ratio of the
  value and density sums is rounded once);
* nrb_refine_control_point_grid vs reg_spline_refineControlPointGrid3D
  (reg-lib/cpu/_reg_localTrans.cpp:1809-2119) onto the next finer reference: every node value
  within 4 float ulps of the reference's (GPU; sums of up to 27 terms weighted 1 to 216), on even and odd dims and a grid whose spacing is
  not a whole number of voxels. The refined values are the same weighted sums (weights 1, 6, 36,
  216 over 8, 32, 128, 512); the reference writes each of its 24 (case, component) sums with
  its own term order, which this kernel does not reproduce, so the last bit differs on a
  quarter of the nodes.
"""
import numpy as np
import pytest

import niftyreg_b200 as nrb
import oracle
from niftyreg_b200 import phantom
from tests.helpers import ensure_built, identity_grid

PYRAMIDS = {
    # (nz, ny, nx), pixdim (dx, dy, dz), origin, levels
    "even": ((64, 80, 96), (1.0, 1.0, 1.0), (0.0, 0.0, 0.0), 3),
    "odd": ((67, 91, 75), (1.0, 1.2, 0.9), (-20.5, 11.0, 3.25), 3),
    "thin_axis": ((40, 130, 129), (0.8, 0.8, 1.5), (5.0, -7.0, 0.0), 3),  # z stops halving
}


def _ref():
    ensure_built()
    if not oracle.ref_available():
        pytest.skip("reference library (oracle/_ref) not built")
    return oracle.Ref()


def _case(name):
    shape, pix, origin, levels = PYRAMIDS[name]
    nz, ny, nx = shape
    img = phantom.blobs_pair(shape, seed=len(name)).reference.astype(np.float32)
    img[0, 0, :3] = np.nan  # NaN voxels travel through the smoothing and the sampling
    xyz = nrb.identity_header(pix, origin)
    return img, (nx, ny, nz), pix, xyz, levels


@pytest.mark.parametrize("name", list(PYRAMIDS))
def test_pyramid_headers_match_reference(name):
    R = _ref()
    img, dim, pix, xyz, levels = _case(name)
    want = R.image_pyramid(img.ravel(), dim, pix, xyz, levels)
    dims, mats, total = nrb.image_pyramid_headers(dim, pix, xyz, levels)
    assert total == sum(int(np.prod(d)) for _, d, _ in want)
    for l, (_, d, m) in enumerate(want):
        assert tuple(dims[l]) == d, (l, dims[l], d)
        assert np.array_equal(mats[l], m), (l, mats[l], m)


@pytest.mark.gpu
@pytest.mark.parametrize("name", list(PYRAMIDS))
def test_pyramid_levels_match_reference(name):
    import torch
    R = _ref()
    img, dim, pix, xyz, levels = _case(name)
    want = R.image_pyramid(img.ravel(), dim, pix, xyz, levels)
    _, _, total = nrb.image_pyramid_headers(dim, pix, xyz, levels)
    out = torch.empty(total, dtype=torch.float32, device="cuda")
    nrb.image_pyramid(torch.from_numpy(img.ravel().copy()).cuda(), dim, pix, xyz, levels, out)
    got = out.cpu().numpy()
    off = 0
    for l, (w, d, _) in enumerate(want):
        n = int(np.prod(d))
        g = got[off:off + n]
        off += n
        w = w.ravel()
        assert np.array_equal(np.isnan(g), np.isnan(w)), l
        ok = ~np.isnan(w)
        err = np.abs(g[ok] - w[ok]).max() / np.abs(w[ok]).max()
        print(f"[pyramid] {name} level {l} {d}: max error {err:.2e} of max, "
              f"{np.mean(g[ok] == w[ok]):.4f} of voxels bit-identical")
        assert err <= 1e-6, (l, err)


def _level64(img, down):
    """One level of the pyramid in double: the normalised Gaussian (sigma 0.7355, radius 2, float
    weights) along x, y and z over the finite values, every `down`-th voxel kept, NaN kept."""
    k = np.exp(-np.arange(-2, 3) ** 2 / (2 * 0.7355 ** 2)) / (0.7355 * 2.506628274631)
    k = k.astype(np.float32).astype(np.float64)
    ok = ~np.isnan(img)
    num, den = np.where(ok, img, 0).astype(np.float64), ok.astype(np.float64)
    for axis in (2, 1, 0):
        num, den = (np.apply_along_axis(lambda a: np.convolve(a, k, "same"), axis, q) for q in (num, den))
    with np.errstate(invalid="ignore", divide="ignore"):
        out = np.where(ok, num / den, np.nan)
    return out[::down[0], ::down[1], ::down[2]]


@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(64, 64, 64), (65, 67, 129), (63, 72, 200), (5, 64, 66)])
def test_pyramid_level_on_tile_edges(shape):
    """One halving at the edges of the smoothing's tiles (32 x 8 outputs, runs along z), axes that
    keep their size, with and without NaN voxels; 1e-6 of the largest magnitude as above. Outputs
    out of a NaN's reach are the same floats with it as without it, and so are all outputs of an
    origin whose coordinates are too large for the fused pass (2^20 mm: still exact, so the
    separate passes sample the same voxels)."""
    import torch
    ensure_built()
    nz, ny, nx = shape
    rng = np.random.default_rng(nz)
    img = rng.normal(300, 100, shape).astype(np.float32)
    bad = img.copy()
    bad[nz // 2, ny // 3, nx // 2] = np.nan
    bad[0, 0, 0] = np.nan
    down = [2 if n // 2 >= 32 else 1 for n in shape]
    got = {}
    for name, data, origin in (("plain", img, 0.0), ("nan", bad, 0.0), ("far", bad, 2.0 ** 20)):
        xyz = nrb.identity_header((1.0, 1.0, 1.0), (origin,) * 3)
        dims, _, total = nrb.image_pyramid_headers((nx, ny, nz), (1.0, 1.0, 1.0), xyz, 2)
        out = torch.empty(total, dtype=torch.float32, device="cuda")
        nrb.image_pyramid(torch.from_numpy(data.ravel()).cuda(), (nx, ny, nz), (1.0, 1.0, 1.0), xyz, 2, out)
        n = int(np.prod(dims[0]))
        got[name] = out.cpu().numpy()[:n].reshape(dims[0][::-1])
        want = _level64(data, down)
        assert got[name].shape == want.shape
        assert np.array_equal(np.isnan(got[name]), np.isnan(want))
        assert np.nanmax(np.abs(got[name] - want)) <= 1e-6 * np.nanmax(np.abs(want)), name
    assert np.array_equal(got["nan"], got["far"], equal_nan=True)
    reach = np.zeros(shape, bool)
    for z, y, x in np.argwhere(np.isnan(bad)):
        reach[max(0, z - 2):z + 3, max(0, y - 2):y + 3, max(0, x - 2):x + 3] = True
    keep = ~reach[::down[0], ::down[1], ::down[2]]
    assert np.array_equal(got["plain"][keep], got["nan"][keep])


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 2, 3, 5, 17, 2049, 1000003])
@pytest.mark.parametrize("offset", [0, 1, 3])
def test_rescale_at_odd_lengths_and_alignments(n, offset):
    """nrb_intensity_rescale against the oracle, bit for bit: lengths around the vector width, bases
    off the 16-byte boundary, NaN values, a constant image (0 / 0), infinite values; the floats on
    either side of the range stay as they were."""
    import torch
    ensure_built()
    O = oracle.Restated()
    rng = np.random.default_rng(n + offset)
    for kind in ("values", "constant", "infinite"):
        img = np.full(n, 3.0, np.float32) if kind == "constant" else rng.normal(0, 500, n).astype(np.float32)
        if kind == "values" and n > 4:
            img[rng.random(n) < 0.1] = np.nan
        if kind == "infinite":
            img[n // 2] = np.inf
        buf = np.full(n + 8, -5.0, np.float32)
        buf[offset:offset + n] = img
        t = torch.from_numpy(buf).cuda()
        nrb.intensity_rescale(t[offset:], n, 2.0, 65.0)
        out = t.cpu().numpy()
        with np.errstate(invalid="ignore"):
            want = O.intensity_rescale(img, 2.0, 65.0)
        assert np.array_equal(out[offset:offset + n], want, equal_nan=True), kind
        assert np.all(out[:offset] == -5.0) and np.all(out[offset + n:] == -5.0)


REFINES = {
    # reference (nz, ny, nx), pixdim, spacing mm at the coarse level
    "even": ((64, 64, 64), (1.0, 1.0, 1.0), 10.0),
    "odd": ((67, 91, 75), (1.0, 1.2, 0.9), 10.0),
    "aniso": ((40, 130, 129), (0.8, 0.8, 1.5), 7.0),
}


@pytest.mark.gpu
@pytest.mark.parametrize("name", list(REFINES))
def test_grid_refinement_matches_reference(name):
    import torch
    R = _ref()
    shape, pix, spacing = REFINES[name]
    nz, ny, nx = shape
    rdim = (nx, ny, nz)
    rxyz = nrb.identity_header(pix, (1.5, -2.0, 0.5))
    # the coarse grid over the reference, displaced, then refined onto the same reference at half
    # the spacing (the registration's refinement onto the next finer level)
    cpp0, cdim, cpix, cxyz = R.create_control_point_grid(rdim, pix, rxyz, (spacing,) * 3)
    rng = np.random.default_rng(len(name))
    cpp = (cpp0 + rng.normal(0, 2.0, cpp0.size)).astype(np.float32)
    want, ndim, npix, nxyz = R.refine_grid(cpp, cdim, cpix, cxyz, rdim, pix, rxyz)
    out = torch.zeros(want.size, dtype=torch.float32, device="cuda")
    nrb.refine_control_point_grid(torch.from_numpy(cpp).cuda(), cdim, out, ndim)
    got = out.cpu().numpy()
    diff = np.abs(got - want)
    # ulps at the scale of the summed node values: a node near the origin is a sum of terms of
    # the order of the grid spacing, whose rounding does not shrink with the result
    ulps = diff / np.spacing(np.maximum(np.abs(want), np.float32(spacing)))
    print(f"[refine] {name}: {tuple(int(v) for v in cdim)} -> {tuple(int(v) for v in ndim)} nodes, "
          f"max |diff| {diff.max():.3g} ({ulps.max():.1f} ulp), {np.mean(got == want):.4f} bit-identical")
    assert ulps.max() <= 4.0
