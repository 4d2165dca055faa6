"""ForwardProjectionROI (Reconstructor.cpp:1519-1529, 649-859) through
esb_rec_forward_projection_roi.

Without CTF the region's rays are exactly the whole-detector projection's
(same kernel, same rays) and nothing else is written. With CTF every slab
image is filtered over the whole detector, so a region's projection spreads
beyond it; the chain is linear in the slab images, so the projections of the
two halves of the detector add up to the whole-detector projection, and a
region covering the detector gives it bit for bit. Traversal lengths are
written for the region's rays only.
"""
import numpy as np
import pytest

from tests.helpers import cuda, host, rel_l2, small_case


def _setup(ctf):
    import artiatomi_b200 as E
    from tests.test_parity_recon import _ctf_cfg

    case = small_case(dims=(48, 40, 20), n_proj=3, W=64, H=56, shift=1.0, psi=0.2)
    W, H, n = case["W"], case["H"], len(case["tilt"])
    cfgd = dict(_ctf_cfg(max(W, H))) if ctf else {}
    defocus = np.tile(np.array([2900.0, 3100.0, 20.0], np.float32), n) if ctf else None
    rec = E.Reconstructor(E.ReconConfig(W, H, n, variant=E.VARIANT_FAST, **cfgd), case["pg"], case["tilt"], defocus)
    vol = cuda(np.ascontiguousarray(case["vol"], np.float32))
    return rec, case, vol, W, H


def _project(rec, case, vol, roi=None, empty=False):
    rec.reset_projections()
    if roi is None:
        rec.forward_projection(case["vg"], vol, 1, empty)
    else:
        rec.forward_projection_roi(case["vg"], vol, 1, roi, empty)
    p, d, _ = rec.views()
    return host(p).copy(), host(d).copy()


@pytest.mark.gpu
@pytest.mark.parametrize("empty", [False, True])
def test_roi_projection_without_ctf_is_the_region_of_the_full_one(empty):
    rec, case, vol, W, H = _setup(False)
    fp, fd = _project(rec, case, vol, empty=empty)
    roi = (9, 5, 41, 30)
    rp, rd = _project(rec, case, vol, roi, empty)
    inside = np.zeros((H, W), bool)
    inside[5:30, 9:41] = True
    np.testing.assert_array_equal(rp[inside], fp[inside])
    np.testing.assert_array_equal(rd[inside], fd[inside])
    assert not rp[~inside].any() and not rd[~inside].any()
    assert np.abs(fd[inside]).max() > 0
    # a region reaching past the detector is clipped; an empty one writes nothing
    cp, cd = _project(rec, case, vol, (-20, 30, W + 50, H + 9), empty)
    np.testing.assert_array_equal(cp[30:], fp[30:])
    np.testing.assert_array_equal(cd[30:], fd[30:])
    ep, ed = _project(rec, case, vol, (20, 20, 20, 40), empty)
    assert not ep.any() and not ed.any()


@pytest.mark.gpu
def test_roi_projection_with_ctf_adds_up_to_the_full_one():
    rec, case, vol, W, H = _setup(True)
    fp, fd = _project(rec, case, vol)
    wp, wd = _project(rec, case, vol, (0, 0, W, H))
    np.testing.assert_array_equal(wp, fp)
    np.testing.assert_array_equal(wd, fd)
    top, tdist = _project(rec, case, vol, (0, 0, W, 23))
    bottom, bdist = _project(rec, case, vol, (0, 23, W, H))
    assert np.abs(top[23:]).max() > 0  # the CTF spreads the region's signal
    assert rel_l2(top + bottom, fp) <= 1e-5, rel_l2(top + bottom, fp)
    np.testing.assert_array_equal(tdist[:23], fd[:23])
    assert not tdist[23:].any()
    np.testing.assert_array_equal(tdist + bdist, fd)


def _noise_case(W, H, nz, psi):
    import artiatomi_b200 as E

    dims, tilt = (W, H, nz), np.array([-40.0, 10.0], np.float32)
    pg = E.projection_geometry(E.Markers(tilt, None, None, None, np.full(2, psi, np.float32)), W, H)
    vol = cuda(np.random.default_rng(2).normal(size=dims[::-1]).astype(np.float32))
    return pg, E.volume_geometry(dims), vol, tilt


@pytest.mark.gpu
@pytest.mark.parametrize("W,H,nz,psi", [(256, 256, 128, 0.2), (160, 158, 96, 0.2), (158, 160, 96, 20.0),
                                        (256, 250, 128, 90.2), (201, 640, 24, 0.0)])
def test_small_regions_of_detectors_that_take_lines_or_runs(W, H, nz, psi):
    """Regions much smaller than a detector whose projection takes lines of 4
    or 2 pixels or rays cut into runs, at offsets inside a line: the whole
    projection's pixels bit for bit, nothing else written."""
    import artiatomi_b200 as E

    pg, vg, vol, tilt = _noise_case(W, H, nz, psi)
    rec = E.Reconstructor(E.ReconConfig(W, H, 2, variant=E.VARIANT_FAST), pg, tilt)
    for i in range(2):
        rec.reset_projections()
        rec.forward_projection(vg, vol, i)
        full = [host(v).copy() for v in rec.views()[:2]]
        assert np.abs(full[0]).max() > 0
        for roi in ((37, 50, 101, 114), (75, 3, 76, 4), (0, 81, W, 98), (2, 0, 141, H)):
            rec.reset_projections()
            rec.forward_projection_roi(vg, vol, i, roi)
            inside = np.zeros((H, W), bool)
            inside[roi[1]:roi[3], roi[0]:roi[2]] = True
            for got, want in zip(rec.views()[:2], full):
                g = host(got)
                np.testing.assert_array_equal(g[inside], want[inside])
                assert not g[~inside].any()


@pytest.mark.gpu
@pytest.mark.parametrize("psi", [0.2, 20.0])
def test_small_regions_with_ctf_add_up(psi):
    """The slab images of 16 regions are those of the whole detector, so that
    their projections add up to its own but for the rounding of the transforms
    and of 16 additions (2e-7 to 3e-7 of the norm; the walk per ray and the
    lines differ by 3e-5)."""
    import artiatomi_b200 as E
    from tests.test_parity_recon import _ctf_cfg

    W = H = 256
    pg, vg, vol, tilt = _noise_case(W, H, 64, psi)
    defocus = np.tile(np.array([2900.0, 3100.0, 20.0], np.float32), 2)
    rec = E.Reconstructor(E.ReconConfig(W, H, 2, variant=E.VARIANT_FAST, **_ctf_cfg(W)), pg, tilt, defocus)

    def projection(roi):
        rec.reset_projections()
        rec.forward_projection_roi(vg, vol, 0, roi)
        return host(rec.views()[0]).astype(np.float64)

    full = projection((0, 0, W, H))
    parts = sum(projection((x, y, x + 64, y + 64)) for x in range(0, W, 64) for y in range(0, H, 64))
    assert rel_l2(parts, full) <= 1e-6, rel_l2(parts, full)
