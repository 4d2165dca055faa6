"""The single-axis forward projector (k_project_axis, k_slicer_axis) where its
layer walk has to go right: volumes thinner than the walk's window, one layer
thick, odd sizes, beams on both sides of 45 degrees (major axis z or x, both
step signs), in-plane rotations at which a warp spans detector rows or
columns, FP32 and 16-bit voxels, and the walk's slabs.

Against the FP64 oracle. The kernel places a ray's samples from its float
start point, ~1e-3 voxel from the oracle's; the volume's gradient is below
0.5 per voxel at an rms of 0.7, so a sum of samples agrees to 1e-3 * 0.5 /
0.7 < 1e-3 of its rms, and to less where the errors of the rays differ:
rel-L2 <= 5e-4. A ray whose length is a whole number of steps to that
accuracy takes one sample more or less, in any 32-bit march (the oracle's
differs from its FP64 one by up to 3.6e-3 here), so a pixel is held to
the nearer of the oracle's two marches.
"""
import numpy as np
import pytest

from tests.helpers import cuda, host, rel_l2

pytestmark = pytest.mark.gpu

TILTS = np.array([0.0, 20.0, -44.9, 45.2, -63.0], np.float32)


def _case(dims, psi, W=26, H=22):
    import artiatomi_b200 as E
    from oracle import geometry as G

    nx, ny, nz = dims
    z, y, x = np.meshgrid(np.arange(nz), np.arange(ny), np.arange(nx), indexing="ij")
    vol = (np.cos(0.4 * x + 0.2 * y) + 0.6 * np.sin(0.3 * z - 0.25 * x + 0.3 * y)).astype(np.float32)
    n = len(TILTS)
    xs, ys = np.linspace(-1.3, 1.1, n).astype(np.float32), np.linspace(0.9, -0.8, n).astype(np.float32)
    ps = np.full(n, psi, np.float32)
    return dict(vol=vol, W=W, H=H, vg=E.volume_geometry(dims), vo=G.volume_geometry(dims),
                pg=E.projection_geometry(E.Markers(TILTS, xs, ys, None, ps), W, H),
                og=G.projection_geometry(TILTS, xs, ys, None, ps, W, H))


@pytest.mark.parametrize("dims", [(3, 5, 2), (4, 9, 1), (1, 6, 7), (33, 17, 5), (5, 8, 40), (70, 12, 9)])
@pytest.mark.parametrize("psi", [0.0, 90.0, 37.0])
def test_axis_projection_small_and_odd(dims, psi):
    import torch

    import artiatomi_b200 as E
    from oracle import driver as D, geometry as G

    c = _case(dims, psi)
    W, H = c["W"], c["H"]
    for i in range(len(TILTS)):
        k = E.set_constant_values(c["pg"][i], c["vg"])
        (p32, _), (p64, do) = [(np.zeros((H, W), np.float32), np.zeros((H, W), np.float32)) for _ in range(2)]
        g = G.orc_geom(c["og"][i], c["vo"])
        D.fp_march(g, c["vol"], 0, W, H, p32, np.zeros((H, W), np.float32), precision=0)
        D.fp_march(g, c["vol"], 0, W, H, p64, do, precision=1)
        for dtype in (torch.float32, torch.float16):
            proj, dist = torch.zeros((H, W), device="cuda"), torch.zeros((H, W), device="cuda")
            E.forward_project(k, cuda(c["vol"]).to(dtype), proj, dist, fast=True)
            # half storage rounds each voxel by up to 2^-11 of its value
            tol = 5e-4 if dtype == torch.float32 else 1e-3
            p = host(proj)
            err = np.linalg.norm(np.minimum(np.abs(p - p64), np.abs(p - p32))) / np.linalg.norm(p64)
            assert err <= tol, (i, dtype, err)
            # entry and exit (|t| ~ 1e4) are rounded to 2^-10 in float
            assert np.abs(host(dist) - do).max() <= 2.5e-3


@pytest.mark.parametrize("dims", [(33, 17, 5), (12, 9, 30)])
@pytest.mark.parametrize("psi", [0.0, 90.0])
def test_axis_slabs_add_up(dims, psi):
    """The slab images of the fused slicer through a reconstructor without
    a CTF effect: every slab's first sample is the one at the ray's start, so
    a slab image is compared with the faithful slicer's, slab by slab, through
    the CTF chain of both variants."""
    import torch

    import artiatomi_b200 as E

    c = _case(dims, psi)
    W, H, n = c["W"], c["H"], len(TILTS)
    defocus = np.tile(np.array([2900.0, 3100.0, 20.0], np.float32), n)
    kw = dict(ctf_mode=True, pixel_size_nm=0.27, ctf_slice_thickness_nm=1.9, ctf_beta_fac=(10.0, 0.0, 0.008, 0.0),
              cut_length=(1.0, 1.0), dim_length=(2.0, 2.0))
    got = []
    for variant in (E.VARIANT_FAST, E.VARIANT_FAITHFUL):
        rec = E.Reconstructor(E.ReconConfig(W, H, n, variant=variant, **kw), c["pg"], TILTS, defocus)
        images = []
        for i in range(n):
            rec.reset_projections()
            rec.forward_projection(c["vg"], cuda(c["vol"]), i)
            torch.cuda.synchronize()
            images.append(host(rec.views()[0]).copy())
        rec.close()
        got.append(np.stack(images))
    assert np.abs(got[1]).max() > 0
    assert rel_l2(got[0], got[1]) <= 5e-4, rel_l2(got[0], got[1])


@pytest.mark.parametrize("dims", [(3, 5, 2), (4, 9, 1), (1, 6, 7), (33, 17, 5), (5, 8, 40)])
@pytest.mark.parametrize("psi", [0.0, 90.0, 37.0])
def test_axis_adjoint_small_and_odd(dims, psi):
    """The gradient kernels' walk: fp_adjoint is the transpose of the loss
    kernel's model, and the loss kernel's volume gradient for zero measured
    values the adjoint of its projection. Both hold to the FP32 rounding of
    the sums (~1e-6 of the Cauchy-Schwarz bound; 1e-5 allowed)."""
    import torch

    import artiatomi_b200 as E

    c = _case(dims, psi)
    x = cuda(c["vol"])
    rng = np.random.default_rng(4)
    for i in range(len(TILTS)):
        k = E.set_constant_values(c["pg"][i], c["vg"])
        for shift in ((0.0, 0.0), (0.7, -1.2)):
            ax = torch.zeros((c["H"], c["W"]), device="cuda")
            grad, out = torch.zeros_like(x), torch.zeros(6, device="cuda", dtype=torch.float64)
            E.projection_loss_grad(k, x, torch.zeros_like(ax), out, shift=shift, grad=grad, proj_out=ax)
            y = cuda(rng.normal(size=tuple(ax.shape)).astype(np.float32))
            aty, atax = torch.zeros_like(x), torch.zeros_like(x)
            E.fp_adjoint(k, aty, y, shift=shift)
            E.fp_adjoint(k, atax, ax, shift=shift)
            lhs, rhs = float((ax.double() * y.double()).sum()), float((x.double() * aty.double()).sum())
            assert abs(lhs - rhs) <= 1e-5 * float(ax.double().norm() * y.double().norm()), (i, shift, lhs, rhs)
            assert rel_l2(host(grad), host(atax)) <= 1e-5, (i, shift)


@pytest.mark.parametrize("dims,W,H", [((389, 97, 7), 101, 397), ((389, 421, 6), 431, 397)])
@pytest.mark.parametrize("psi", [0.0, 0.1, 0.3, -0.29, 90.2, 179.6])
def test_lines_of_rays(dims, W, H, psi):
    """Next to no in-plane rotation: k_project_planes and k_slicer_planes
    (2 pixels per thread on the small detector, 4 on the large one at no or
    0.1 degrees, 2 on either or the walk per ray at the others) against the faithful march and slicer over
    the same voxels, for every voxel type, a detector region and slabs; the
    bound as above, of which the lines' expansion takes a tenth."""
    import torch

    import artiatomi_b200 as E

    c = _case(dims, psi, W, H)
    n = len(TILTS)
    roi = (3, 5, W - 4, H - 1)
    for i in range(n):
        k = E.set_constant_values(c["pg"][i], c["vg"])
        for dtype in (torch.float32, torch.float16, torch.bfloat16):
            vol = cuda(c["vol"]).to(dtype)
            (p, d), (q, e), (r, s) = [[torch.full((H, W), 0.25, device="cuda") for _ in range(2)] for _ in range(3)]
            E.forward_project(k, vol, p, d, fast=True)
            E.forward_project(k, vol, q, e)
            E.forward_project(k, vol, r, s, roi=roi, fast=True)
            torch.cuda.synchronize()
            p, d, q, e, r, s = (host(t) for t in (p, d, q, e, r, s))
            assert rel_l2(p - 0.25, q - 0.25) <= 5e-4, (i, dtype, rel_l2(p - 0.25, q - 0.25))
            assert np.array_equal(d, e)
            inside = np.zeros((H, W), bool)
            inside[roi[1]:roi[3], roi[0]:roi[2]] = True
            assert np.all(r[~inside] == 0.25) and np.all(s[~inside] == 0.25)
            assert rel_l2(r[inside] - 0.25, q[inside] - 0.25) <= 5e-4 and np.array_equal(s[inside], e[inside])
    defocus = np.tile(np.array([2900.0, 3100.0, 20.0], np.float32), n)
    kw = dict(ctf_mode=True, pixel_size_nm=0.27, ctf_slice_thickness_nm=1.9, ctf_beta_fac=(10.0, 0.0, 0.008, 0.0),
              cut_length=(1.0, 1.0), dim_length=(2.0, 2.0))
    got = []
    for variant in (E.VARIANT_FAST, E.VARIANT_FAITHFUL):
        rec = E.Reconstructor(E.ReconConfig(W, H, n, variant=variant, **kw), c["pg"], TILTS, defocus)
        rec.reset_projections()
        rec.forward_projection(c["vg"], cuda(c["vol"]), 2)
        torch.cuda.synchronize()
        got.append(host(rec.views()[0]).copy())
        rec.close()
    assert np.abs(got[1]).max() > 0
    assert rel_l2(got[0], got[1]) <= 5e-4, rel_l2(got[0], got[1])


@pytest.mark.parametrize("dims", [(3, 5, 2), (4, 9, 1), (33, 17, 5), (5, 8, 40)])
@pytest.mark.parametrize("phi,tilt_x", [(0.02, 0.0), (0.8, 0.0), (0.0, 13.5)])
def test_declined_beam_small_and_odd(dims, phi, tilt_x):
    """tilted_sum: rays whose y moves slowly, by nearly nothing and by up to
    nearly a quarter of a layer per layer (13.5 degrees about the tilt axis'
    normal; the series' projections beyond take the walk from cell to cell),
    against the nearer of the oracle's marches (above)."""
    import torch

    import artiatomi_b200 as E
    from oracle import driver as D, geometry as G

    W, H, n = 26, 22, len(TILTS)
    c = _case(dims, 0.0, W, H)
    psi = np.linspace(-9.0, 11.0, n).astype(np.float32)
    pg = E.projection_geometry(E.Markers(TILTS, None, None, None, psi), W, H, E.TiltConfig(phi_angle=phi, add_tilt_x_angle=tilt_x))
    og = G.projection_geometry(TILTS, None, None, None, psi, W, H,
                               cfg={"phi_angle": phi, "add_tilt_x_angle": tilt_x})
    for i in range(n):
        k = E.set_constant_values(pg[i], c["vg"])
        g = G.orc_geom(og[i], c["vo"])
        marches = []
        for precision in (0, 1):
            p = np.zeros((H, W), np.float32)
            D.fp_march(g, c["vol"], 0, W, H, p, np.zeros_like(p), precision=precision)
            marches.append(p)
        for dtype, tol in ((torch.float32, 5e-4), (torch.float16, 1e-3)):
            proj, dist = torch.zeros((H, W), device="cuda"), torch.zeros((H, W), device="cuda")
            E.forward_project(k, cuda(c["vol"]).to(dtype), proj, dist, fast=True)
            d = [np.abs(host(proj) - p) for p in marches]
            err = np.linalg.norm(np.minimum(*d)) / np.linalg.norm(marches[1])
            assert err <= tol, (i, dtype, err)


@pytest.mark.parametrize("dims,W,H", [((40, 24, 12), 48, 44), ((96, 40, 30), 60, 100)])
@pytest.mark.parametrize("psi", [0.0, 25.0, 90.0])
def test_nan_voxels_at_the_faces(dims, W, H, psi):
    """A NaN voxel at the volume's faces reaches every ray of the faithful march
    that interpolates it, and others only where a layer or a cell of the walk
    holds no sample (its voxels then have a weight of 0, which is NaN too):
    rays that pass a corner, 1 in 6.7 (the samples of a voxel's length), so at
    most a fifth more. Reads of the window's outer positions without a crossing
    give a quarter to a third more."""
    import torch

    import artiatomi_b200 as E

    n = len(TILTS)
    pg = E.projection_geometry(E.Markers(TILTS, None, None, None, np.full(n, psi, np.float32)), W, H)
    vg = E.volume_geometry(dims)
    clean = np.random.default_rng(0).normal(size=dims[::-1]).astype(np.float32)
    at = [(0, dims[1] // 2, 3), (dims[2] - 1, 3, dims[0] - 2), (1, dims[1] // 3, dims[0] - 1), (dims[2] - 2, 8, 0)]
    extra = exact = 0
    for i in range(n):
        k = E.set_constant_values(pg[i], vg)
        for p in at:
            vol = clean.copy()
            vol[p] = np.nan
            masks = []
            for fast in (False, True):
                proj, dist = torch.zeros((H, W), device="cuda"), torch.zeros((H, W), device="cuda")
                E.forward_project(k, cuda(vol), proj, dist, fast=fast)
                masks.append(~np.isfinite(host(proj)))
            assert not (masks[0] & ~masks[1]).any()
            extra += int((masks[1] & ~masks[0]).sum())
            exact += int(masks[0].sum())
    assert exact > 0 and extra <= 0.2 * exact, (extra, exact)


@pytest.mark.parametrize("psi", [0.05, 0.13, 0.27, 0.4])
def test_lines_are_as_exact_as_the_walk(psi):
    """Lines of rays against the walk per ray on white noise, beams from 0
    degrees on: the same rays on a detector too narrow for lines. Rays of a line
    lie up to e = 1/144 voxel from its middle ray; a sample that this carries
    across a face is off by at most e times the kink there, whose variance is
    2.7 of the noise's. 2 e / 0.13 of the layers have one, with e^2 / 3 on
    average, against a projection of variance 0.44 / 0.13^2 per layer: 0.5
    e^1.5 at the line's ends, half of it over its rays, 1.5e-4."""
    import torch

    import artiatomi_b200 as E

    dims, W, H = (389, 421, 48), 397, 431
    tilts = np.array([0.0, 1.5, 6.0, 14.0, -33.0, 58.0], np.float32)
    pg = E.projection_geometry(E.Markers(tilts, None, None, None, np.full(len(tilts), psi, np.float32)), W, H)
    vg = E.volume_geometry(dims)
    vol = cuda(np.random.default_rng(0).normal(size=dims[::-1]).astype(np.float32))
    for i in range(len(tilts)):
        k = E.set_constant_values(pg[i], vg)
        lines, dist = torch.zeros((H, W), device="cuda"), torch.zeros((H, W), device="cuda")
        E.forward_project(k, vol, lines, dist, fast=True)
        walk, dist = torch.zeros((H, 16), device="cuda"), torch.zeros((H, 16), device="cuda")
        E.forward_project(k, vol, walk, dist, fast=True)
        a, b = host(lines)[:, :16], host(walk)
        assert np.abs(b).max() > 0
        assert rel_l2(a, b) <= 1.5e-4, (i, rel_l2(a, b))
