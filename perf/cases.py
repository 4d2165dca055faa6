"""Performance cases of the EmSART path: what a reconstruction program has this framework do.

A case names one operation with its sizes and options. Six operations cover the path:

* ``sart``     one further SART iteration on a running reconstruction (forward projection, compare, back-projection
               for every projection of the series), through ``Reconstructor.sart``;
* ``project``  forward projections of a volume over a tilt series, through ``Reconstructor.forward_projection``;
* ``subvol``   the weighted back-projection of particle boxes, through ``Reconstructor.subvolume_wbp``;
* ``loss``     the projection loss with its volume and shift gradients, through ``projection_loss_grad``;
* ``refine``   shift measurements of a particle (region projections, compare, cross-correlation), through the
               reconstructor's calls of EmSartRefine;
* ``prepare``  raw projections to normalised images, through ``Reconstructor.prepare_projection``.

``exact`` states each operation in plain torch in 64 bits.
"""
import math

import numpy as np
import torch

import artiatomi_b200 as E
from artiatomi_b200 import _lib as L

DISTANCE = -10000.0  # detector plane, voxels from the origin
PIXEL_NM, SLAB_NM, CS_MM, KV, WIENER = 0.27, 30.0, 2.7, 300.0, 0.1
DTYPES = {"f32": torch.float32, "f16": torch.float16, "bf16": torch.bfloat16}


def series(op, nx, ny, nz, W, H, n, *, sirt=1, os=1, ctf=False, dtype="f32", psi=0.0, jitter=0.0, shift=0.0, phi=0.0,
           aniso=1.0):
    """A tilt series on a volume. psi: in-plane rotation of the tilt axis (degrees) with its jitter; shift: alignment
    shifts U(+-shift) pixels; phi: declination of the beam against the tilt axis (degrees); aniso: magnification
    anisotropy."""
    return dict(op=op, nx=nx, ny=ny, nz=nz, W=W, H=H, n=n, sirt=sirt, os=os, ctf=ctf, dtype=dtype, psi=psi,
                jitter=jitter, shift=shift, phi=phi, aniso=aniso)


def listed():
    return [
        # a crop or a binned preview: small kernels one after the other, launches count
        dict(series("sart", 64, 64, 32, 64, 64, 9, shift=1.0, jitter=0.2), name="sart_preview"),
        # a binned tomogram without CTF, the plain SART configuration of the benchmark
        dict(series("sart", 256, 256, 128, 256, 256, 41), name="sart_plain"),
        # a cropped region with 3-D CTF, aligned per tilt
        dict(series("sart", 256, 256, 64, 256, 256, 61, sirt=4, os=2, ctf=True, shift=2.0, jitter=0.3),
             name="sart_ctf"),
        # the size of the headline benchmark (1024 x 1024 x 256, 3-D CTF), a part of its tilts
        dict(series("sart", 1024, 1024, 256, 1024, 1024, 16, sirt=4, os=2, ctf=True, shift=2.0, jitter=0.3),
             name="sart_ctf_large"),
        # a volume stored in 16 bits, large subsets
        dict(series("sart", 512, 512, 128, 512, 512, 16, sirt=8, os=2, ctf=True, dtype="f16", shift=2.0, jitter=0.3),
             name="sart_half"),
        # a stack as the microscope gave it: the tilt axis runs across the image, odd sizes, rectangular detector
        dict(series("project", 509, 381, 97, 493, 517, 5, psi=84.3, shift=3.0, jitter=0.3), name="project_rotated"),
        # an alignment with beam declination and magnification anisotropy
        dict(series("sart", 256, 240, 96, 272, 256, 13, sirt=2, os=2, shift=2.0, jitter=0.3, phi=0.8, aniso=1.012),
             name="sart_declined"),
        # particle boxes of three sizes out of CTF-corrected projections
        dict(series("subvol", 1024, 1024, 300, 1024, 1024, 9, os=2, ctf=True), particles=200, name="subvol_ctf"),
        # the same from plain weighted projections, many tilts
        dict(series("subvol", 1024, 1024, 300, 1024, 1024, 41), particles=60, name="subvol_plain"),
        # gradients of the volume and of the alignment
        dict(series("loss", 512, 512, 128, 512, 512, 3), name="loss_gradients"),
        # shift refinement of one particle over a few tilts
        dict(series("refine", 512, 512, 160, 512, 512, 3, ctf=True, shift=2.0, jitter=0.3), box=64, name="refine_ctf"),
        # raw camera frames (rectangular) to normalised projections
        dict(op="prepare", W=1920, H=1440, n=3, raw="int16", name="prepare_int16"),
    ]


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    op = rng.choice(["sart", "sart", "sart", "sart", "project", "subvol", "loss", "refine", "prepare"])
    if op == "prepare":
        W = log_int(64, 2048)
        return dict(op=op, W=W, H=int(W * rng.uniform(0.6, 1.0)), n=rng.randint(1, 5),
                    raw=rng.choice(["int16", "uint16", "float32"]))
    nx, ny, nz = log_int(48, 640), log_int(48, 640), log_int(16, 160)
    if op == "refine":  # about square: the correlation pads the detector to a square
        ny = int(nx * rng.uniform(0.7, 1.4))
    # without in-plane rotation the tilt axis (y of the volume) runs along the detector's rows
    W, H = int(ny * rng.uniform(0.85, 1.15)), int(nx * rng.uniform(0.85, 1.15))
    c = series(op, nx, ny, nz, W, H, rng.randint(3, 12), shift=rng.choice([0.0, 2.0]), jitter=rng.choice([0.0, 0.3]))
    if op in ("sart", "project"):
        c.update(sirt=rng.choice([1, 2, 3, 4, 8]), os=rng.choice([1, 2, 2]), ctf=rng.random() < 0.5,
                 dtype=rng.choice(["f32", "f32", "f32", "f16", "bf16"]))
        if rng.random() < 0.3:
            c.update(psi=rng.uniform(-180.0, 180.0))
        if rng.random() < 0.2:
            c.update(phi=rng.uniform(-1.5, 1.5))
        if rng.random() < 0.2:
            c.update(aniso=rng.uniform(0.98, 1.02))
    if op == "subvol":
        c.update(nx=nx + 64, ny=ny + 64, nz=nz + 64, W=W + 64, H=H + 64, os=rng.choice([1, 2]), ctf=rng.random() < 0.5,
                 particles=log_int(1, 200))
    if op == "loss":
        c.update(n=rng.randint(1, 3))
    if op == "refine":
        c.update(nx=nx + 64, ny=ny + 64, nz=nz + 64, W=W // 2 * 2 + 64, H=H // 2 * 2 + 64, n=rng.randint(1, 4), shift=2.0, jitter=0.3,
                 ctf=rng.random() < 0.5, box=rng.choice([32, 48, 64]))
    return c


# ------------------------------------------------------------------ inputs
def _device():
    return torch.device("cuda")


def _generator(seed):
    return torch.Generator(device=_device()).manual_seed(int(seed))


def _density(shape, gen, grain=8):
    """Smooth density with contrast at several voxels' scale, and weak noise."""
    low = tuple(max(2, -(-s // grain)) for s in shape)
    v = torch.randn((1, 1) + low, generator=gen, device=_device())
    v = torch.nn.functional.interpolate(v, size=shape, mode="trilinear" if len(shape) == 3 else "bilinear",
                                        align_corners=True)[0, 0]
    return v + 0.1 * torch.randn(shape, generator=gen, device=_device())


def _images(case, gen, count, noise=1.0):
    """Normalised projections: smooth signal under noise, low-passed as preparation leaves them."""
    H, W = case["H"], case["W"]
    out = []
    for _ in range(count):
        img = _density((H + 2, W + 2), gen)
        img = img + (8.0 / 3.0) * noise * torch.randn((H + 2, W + 2), generator=gen, device=_device())
        img = 0.25 * img[:-2] + 0.5 * img[1:-1] + 0.25 * img[2:]
        out.append(0.25 * img[:, :-2] + 0.5 * img[:, 1:-1] + 0.25 * img[:, 2:])
    return torch.stack(out)


def _alignment(case, seed):
    """Tilt angles, shifts and psi of the series, and the defocus table."""
    n = case["n"]
    rng = np.random.default_rng(int(seed))
    tilt = np.linspace(-60.0, 60.0, n).astype(np.float32) if n > 1 else np.array([20.0], np.float32)
    xs = rng.uniform(-case["shift"], case["shift"], n).astype(np.float32)
    ys = rng.uniform(-case["shift"], case["shift"], n).astype(np.float32)
    psi = (case["psi"] + rng.uniform(-case["jitter"], case["jitter"], n)).astype(np.float32)
    mid = rng.uniform(2500.0, 3500.0, n)
    defocus = np.stack([mid - 50.0, mid + 50.0, rng.uniform(0.0, 180.0, n)], 1).astype(np.float32)
    return tilt, xs, ys, psi, defocus


def _beta(case):
    """CTFBetaFac: the envelope, and no correction below this radius of the N x N transform."""
    return (200.0 if max(case["W"], case["H"]) >= 1024 else 10.0, 0.0, 0.008, 0.0)


def _anisotropy(case):
    """Magnification anisotropy matrix (35 degrees) and its inverse, None without."""
    if case["aniso"] == 1.0:
        return None, None
    a = np.float32(case["aniso"])
    return (E.mag_aniso_matrix(float(a), 35.0, case["W"], case["H"]),
            E.mag_aniso_matrix(float(np.float32(1.0) / a), 35.0, case["W"], case["H"]))


def _reconstructor(case, seed):
    tilt, xs, ys, psi, defocus = _alignment(case, seed)
    pg = E.projection_geometry(E.Markers(tilt, xs, ys, None, psi), case["W"], case["H"],
                               E.TiltConfig(phi_angle=case["phi"]))
    kw = {}
    if case["ctf"]:
        kw = dict(ctf_mode=True, pixel_size_nm=PIXEL_NM, cs_mm=CS_MM, voltage_kv=KV, amp_contrast=0.0,
                  ctf_slice_thickness_nm=SLAB_NM, ctf_beta_fac=_beta(case), wiener_noise_level=WIENER)
    cfg = E.ReconConfig(case["W"], case["H"], case["n"], lambda_=0.5, oversampling=case["os"], cut_length=(10.0, 10.0),
                        dim_length=(20.0, 20.0), variant=E.VARIANT_FAST, **kw)
    mag, inv = _anisotropy(case)
    return E.Reconstructor(cfg, pg, tilt, defocus.ravel() if case["ctf"] else None, mag, inv), pg


def _particles(case, seed):
    """Box sizes, positions (1-based voxels) and per-tilt extra shifts."""
    rng = np.random.default_rng(int(seed) + 1)
    P, dims = case["particles"], (case["nx"], case["ny"], case["nz"])
    sizes = np.random.default_rng(1).choice([48, 64, 96], size=P, p=[0.5, 0.35, 0.15])
    sizes = np.minimum(sizes, 4 * (min(dims) // 4))
    pos = np.stack([rng.uniform(sizes / 2, d - sizes / 2) for d in dims], 1).astype(np.float32)
    return sizes, pos, rng.uniform(-1.5, 1.5, (P, case["n"], 2)).astype(np.float32)


def _refinement(case, seed):
    """Particle position (1-based), its Euler angles and per tilt the detector region around it."""
    rng = np.random.default_rng(int(seed) + 1)
    dims, box = (case["nx"], case["ny"], case["nz"]), case["box"]
    pos = np.array([rng.uniform(box / 2 + 2, d - box / 2 - 1) for d in dims], np.float32)
    safe = 100 + 2 * box + 2 * 10
    tilt, xs, ys, psi, _ = _alignment(case, seed)
    rois = []
    for f in _frames(case, seed):
        c = pos - 0.5 - np.array(dims) / 2.0
        x, y, _ = f["to_detector"] @ (c - f["det"])
        rois.append((max(int(x) - safe, 0), max(int(y) - safe, 0), int(x) + safe, int(y) + safe))
    return pos, rng.uniform(0.0, 360.0, 3).astype(np.float32), rois


def _raw_frames(case, gen):
    """Camera counts with gradients and a few hot pixels."""
    H, W = case["H"], case["W"]
    y, x = torch.meshgrid(torch.arange(H, device=_device()), torch.arange(W, device=_device()), indexing="ij")
    out = []
    for _ in range(case["n"]):
        img = 200.0 + 40.0 * torch.sin(x / 70.0) + 30.0 * torch.cos(y / 50.0)
        img = torch.poisson(img, generator=gen)
        hot = torch.randint(0, H * W, (6,), generator=gen, device=_device())
        img.view(-1)[hot] = 5000.0
        out.append(img.to(torch.float32) * 0.37 if case["raw"] == "float32" else img.to(getattr(torch, case["raw"])))
    return torch.stack([o.view(torch.int16) for o in out]).view(torch.uint16) if case["raw"] == "uint16" else \
        torch.stack(out)


FILTER = dict(normalization=1, correct_bad_pixels=1, bad_pixel_value=10.0, lp=300.0, hp=4.0, lps=30.0, hps=2.0)


def prepare(case, seed):
    gen = _generator(seed)
    if case["op"] == "prepare":
        cfg = E.ReconConfig(case["W"], case["H"], case["n"], variant=E.VARIANT_FAST)
        pg = E.projection_geometry(E.Markers(np.zeros(case["n"], np.float32)), case["W"], case["H"])
        return dict(case=case, raw=_raw_frames(case, gen), rec=E.Reconstructor(cfg, pg, np.zeros(case["n"])),
                    out=torch.empty((case["n"], case["H"], case["W"]), device=_device()))
    rec, pg = _reconstructor(case, seed)
    shape = (case["nz"], case["ny"], case["nx"])
    s = dict(case=case, rec=rec, pg=pg, vg=E.volume_geometry((case["nx"], case["ny"], case["nz"])))
    if case["op"] == "sart":
        s["start"] = _density(shape, gen).to(DTYPES[case["dtype"]])
        s["vol"] = torch.empty_like(s["start"])
        s["projections"] = _images(case, gen, case["n"])
        s["order"] = _order(case, seed)
    elif case["op"] == "project":
        s["vol"] = _density(shape, gen).to(DTYPES[case["dtype"]])
        s["out"] = torch.empty((2, case["n"], case["H"], case["W"]), device=_device())
        s["views"] = rec.views()
    elif case["op"] == "subvol":
        sizes, pos, extra = _particles(case, seed)
        tilt, xs, ys, psi, _ = _alignment(case, seed)
        s["sub"] = [E.subvolume_geometry(int(z), 1.0, s["vg"], p) for z, p in zip(sizes, pos)]
        s["pairs"] = (L.ProjGeom * (len(sizes) * case["n"]))()
        for p in range(len(sizes)):
            g = E.projection_geometry(E.Markers(tilt, xs, ys, None, psi), case["W"], case["H"], extra_shift=extra[p])
            s["pairs"][p * case["n"]:(p + 1) * case["n"]] = list(g)
        s["boxes"] = [torch.zeros((int(z),) * 3, device=_device()) for z in sizes]
        s["projections"] = _images(case, gen, case["n"])
        s["order"] = np.arange(case["n"], dtype=np.int32)
    elif case["op"] == "loss":
        s["vol"] = _density(shape, gen)
        s["measured"] = _images(case, gen, case["n"], noise=5.0)
        s["shifts"] = np.random.default_rng(int(seed) + 2).uniform(-1.0, 1.0, (case["n"], 2))
        s["constants"] = [E.set_constant_values(pg[i], s["vg"]) for i in range(case["n"])]
        s["grad"] = torch.empty(shape, device=_device())
        s["sums"] = torch.empty((case["n"], 6), dtype=torch.float64, device=_device())
    else:
        pos, angles, rois = _refinement(case, seed)
        s["vol"] = _density(shape, gen)
        s["measured"] = _images(case, gen, case["n"])
        s["model"] = _density((case["box"],) * 3, gen)
        s["sub"] = E.subvolume_geometry(case["box"], 1.0, s["vg"], pos)
        s["rotation"], s["rois"] = E.rotation_matrix(*angles), rois
        s["rotated"] = torch.empty_like(s["model"])
        s["residual"] = torch.empty((case["n"], case["H"], case["W"]), device=_device())
        s["maps"] = torch.empty((case["n"], 40, 40), device=_device())
        s["views"] = rec.views()
        rec.forward_projection(s["vg"], s["vol"], 0)  # the whole reconstruction once, as a look at the alignment
    return s


def _order(case, seed):
    order = np.random.default_rng(int(seed) + 2).permutation(case["n"])
    return np.ascontiguousarray(order, np.int32)


# ------------------------------------------------------------------ the pass
def run(s):
    case = s["case"]
    rec = s["rec"]
    if case["op"] == "sart":
        s["vol"].copy_(s["start"])
        rec.sart(s["vg"], s["vol"], s["projections"], s["order"], iterations=1, sirt_count=case["sirt"],
                 volume_is_empty=False)
        return s["vol"]
    if case["op"] == "project":
        image, length, _ = s["views"]
        for i in range(case["n"]):
            rec.reset_projections()
            rec.forward_projection(s["vg"], s["vol"], i)
            s["out"][0, i].copy_(image)
            s["out"][1, i].copy_(length)
        return s["out"]
    if case["op"] == "subvol":
        for b in s["boxes"]:
            b.zero_()
        rec.subvolume_wbp(s["vg"], s["sub"], s["pairs"], s["boxes"], s["projections"], s["order"])
        return torch.cat([b.view(-1) for b in s["boxes"]])
    if case["op"] == "loss":
        s["grad"].zero_()
        s["sums"].zero_()
        for i in range(case["n"]):
            E.projection_loss_grad(s["constants"][i], s["vol"], s["measured"][i], s["sums"][i],
                                   shift=tuple(s["shifts"][i]), grad=s["grad"])
        return dict(sums=s["sums"], grad=s["grad"])
    if case["op"] == "refine":
        image = s["views"][0]
        E.rotate_volume(s["model"], s["rotated"], s["rotation"])
        found, peaks = [], []
        for i in range(case["n"]):
            rec.reset_projections()
            rec.forward_projection_roi(s["vg"], s["vol"], i, s["rois"][i])
            rec.compare(s["vg"], s["measured"][i], i)
            s["residual"][i].copy_(image)
            rec.reset_projections()
            rec.forward_projection_roi(s["sub"], s["rotated"], i, s["rois"][i])
            shift, peak = rec.cc_displacement(s["residual"][i], image, 10, cc_map=s["maps"][i])
            found.append([int(v) for v in shift])
            peaks.append(peak)
        return dict(residual=s["residual"], maps=s["maps"], shifts=np.array(found), peaks=np.array(peaks))
    stats = [rec.prepare_projection(s["raw"][i], s["out"][i], **FILTER) for i in range(case["n"])]
    return dict(images=s["out"], stats=np.array([t[:2] for t in stats]), bad=np.array([t[2] for t in stats]))


def work(case):
    """Volume, box and image bytes each touched once per ordered subset (a subset's projections can share them), and the
    floating-point operations of the projection model: per ray and layer two cells of the interpolation lattice, per
    voxel and back-projected image the sub-pixel samples of its shadow."""
    img = 4.0 * case["W"] * case["H"]
    pixels = float(case["W"] * case["H"])
    n = case["n"]
    if case["op"] == "prepare":
        side = max(case["W"], case["H"])
        raw = pixels * (4 if case["raw"] == "float32" else 2)
        return dict(bytes=n * (raw + img), flops=n * 2 * 2.5 * side * side * 2 * math.log2(side))
    voxels = float(case["nx"] * case["ny"] * case["nz"])
    size = 4.0 if case["dtype"] == "f32" else 2.0
    side = max(case["W"], case["H"])
    fft = 2 * 2.5 * side * side * 2 * math.log2(side) if case["ctf"] else 0.0
    forward = 4 * 30 * pixels * case["nz"] * 1.4  # 4 rays a pixel, layers along the tilted ray
    backward = voxels * 12 * 1.5 * case["os"] ** 2
    if case["op"] == "sart":
        subsets = -(-n // case["sirt"])
        slabs = 1.0 + 1.4 * case["nz"] * PIXEL_NM / SLAB_NM if case["ctf"] else 0.0
        return dict(bytes=subsets * 3 * voxels * size + n * 2 * img, flops=n * (forward + backward + 2 * slabs * fft))
    if case["op"] == "project":
        return dict(bytes=voxels * size + n * 2 * img, flops=n * (forward + fft))
    if case["op"] == "subvol":
        box = case["particles"] * 66.0 ** 3
        return dict(bytes=8 * box + n * img, flops=n * (box * 12 * 1.5 * case["os"] ** 2 + 5 * fft))
    if case["op"] == "loss":
        return dict(bytes=3 * 4 * voxels + n * img, flops=n * 3 * forward)
    region = min(1.0, (2.0 * (120 + 2 * case["box"])) ** 2 / pixels)
    return dict(bytes=4 * voxels * region + n * 5 * img, flops=n * (region * forward + 3 * fft + 2.5 * side * side))


def tolerance(case):
    """About four times the error against 64 bits that was measured over the ranges. The largest single differences are
    voxels and pixels at which a sample lies on the edge of a shadow, a slab or a ray's end and is taken or not; an
    in-plane rotation of the detector or a declined beam has more of them."""
    op = case["op"]
    if op == "prepare":
        return {"rel": 8e-6}
    if op == "project":
        return {"rel": 1.5e-4, "max": 0.02}
    if op == "sart":
        rel = {"f32": 3e-4, "f16": 1.5e-3, "bf16": 1e-2}[case["dtype"]]
        return {"rel": max(rel, 2e-3) if case["psi"] or case["phi"] else rel, "max": 0.5}
    return {"subvol": {"rel": 3e-3, "max": 0.99}, "loss": {"rel": 3e-3, "max": 0.5},
            "refine": {"rel": 2e-3, "max": 0.2}}[op]


# ------------------------------------------------------------------ the same in 64 bits
F64 = torch.float64


def _rotation(axis, degrees):
    a = math.radians(degrees)
    c, s = math.cos(a), math.sin(a)
    return {"x": np.array([[1, 0, 0], [0, c, -s], [0, s, c]]), "y": np.array([[c, 0, s], [0, 1, 0], [-s, 0, c]]),
            "z": np.array([[c, -s, 0], [s, c, 0], [0, 0, 1]])}[axis]


def _frames(case, seed, extra=None):
    """Detector frames as the alignment defines them, in the 32-bit numbers that a program passes on."""
    tilt, xs, ys, psi, _ = _alignment(case, seed)
    W, H = case["W"], case["H"]
    f32 = np.float32
    out = []
    for i in range(case["n"]):
        phi = _rotation("x", float(f32(case["phi"])))
        m = phi @ _rotation("y", float(tilt[i])) @ phi.T @ _rotation("z", -float(psi[i])) @ \
            np.array([[0.0, -1, 0], [1, 0, 0], [0, 0, -1]])
        u, v = m[:, 0].astype(f32), m[:, 1].astype(f32)
        sx, sy = f32(xs[i]), f32(ys[i])
        if extra is not None:
            sx, sy = f32(sx + extra[i][0]), f32(sy + extra[i][1])
        det = (m @ np.array([-0.5 * W, -0.5 * H, DISTANCE])).astype(f32) - u * sx - v * sy
        n = -np.cross(u, v)
        n = (n * f32(1.0 / math.sqrt(float(n @ n)))).astype(f32)
        frame = np.stack([u, v, n], 1).astype(np.float64)
        out.append(dict(u=u.astype(np.float64), v=v.astype(np.float64), n=n.astype(np.float64),
                        det=det.astype(np.float64), to_detector=np.linalg.inv(frame), tilt=float(tilt[i])))
    return out


def _place(dims, lo=None):
    """A volume in space: lower corner, size; voxels of size 1."""
    d = np.array(dims, np.float64)
    return dict(dims=tuple(int(v) for v in dims), lo=-0.5 * d if lo is None else np.asarray(lo, np.float64), size=d)


def _slabs(f, whole):
    """Boundaries of the defocus slabs along the beam."""
    corners = [whole["lo"] + whole["size"] * np.array([x, y, z]) for x in (0, 1) for y in (0, 1) for z in (0, 1)]
    t = [float(f["n"] @ (c - f["det"])) for c in corners]
    bounds = [min(t)]
    while bounds[-1] < max(t):
        bounds.append(bounds[-1] + SLAB_NM / PIXEL_NM)
    return bounds


def _project64(vol, f, place, W, H, mag, roi=None, bounds=None):
    """Mean over 2 x 2 rays of a pixel of the sampled line integrals (one image per slab with `bounds`), and the rays'
    mean length. Samples lie every 0.15 voxels, on the 32-bit grid of the ray parameter; a slab's first sample is read
    at the ray's start on the detector."""
    dev = vol.device
    lo, size = torch.tensor(place["lo"], device=dev), torch.tensor(place["size"], device=dev)
    det, u, v, n = (torch.tensor(f[k], device=dev) for k in ("det", "u", "v", "n"))
    x0, y0, x1, y1 = (0, 0, W, H) if roi is None else (max(roi[0], 0), max(roi[1], 0), min(roi[2], W), min(roi[3], H))
    count = 1 if bounds is None else len(bounds) - 1
    out = torch.zeros((count, H, W), dtype=F64, device=dev)
    length = torch.zeros((H, W), dtype=F64, device=dev)
    step = round(0.15 * 1024) / 1024
    last = size - 1

    def sample(p):
        q = torch.minimum(torch.clamp(p - lo - 0.5, min=0.0), last)
        g = 2.0 * q / torch.clamp(last, min=1.0) - 1.0
        return torch.nn.functional.grid_sample(vol[None, None], g[None, None], mode="bilinear", padding_mode="border",
                                               align_corners=True)[0, 0, 0]

    def chord(px, py):
        ax, ay = mag[0] * px + mag[1] * py + mag[2], mag[3] * px + mag[4] * py + mag[5]
        s = det + ax[..., None] * u + ay[..., None] * v
        a, b = (lo - s) / n, (lo + size - s) / n
        # (a beam along an axis crosses the other pairs of faces nowhere, or everywhere)
        a, b = torch.nan_to_num(a, nan=-1e30), torch.nan_to_num(b, nan=1e30)
        return s, torch.minimum(a, b).amax(-1), torch.maximum(a, b).amin(-1)

    xx = torch.arange(x0, x1, device=dev, dtype=F64)
    rows = max(1, 20000 // max(1, x1 - x0))
    for r0 in range(y0, y1, rows):
        yy = torch.arange(r0, min(r0 + rows, y1), device=dev, dtype=F64)
        hits = torch.zeros((len(yy), len(xx)), dtype=F64, device=dev)
        total = torch.zeros_like(hits)
        for ox, oy in ((0.25, 0.25), (0.25, 0.75), (0.75, 0.25), (0.75, 0.75)):
            py, px = torch.meshgrid(yy + oy, xx + ox, indexing="ij")
            s, tin, tout = chord(px, py)
            hit = tout > tin
            hits += hit
            total += torch.where(hit, tout - tin, torch.zeros_like(tin))
            for k in range(count):
                t0, t1 = tin, tout
                if bounds is not None:
                    t0, t1 = torch.clamp(tin, min=bounds[k]), torch.clamp(tout, max=bounds[k + 1])
                some = hit & (t0 <= t1)
                if not bool(some.any()):
                    continue
                src, start = s[some], t0[some]
                J = torch.floor((t1[some] - start) / step) + 1
                acc = torch.zeros_like(start)
                block = max(1, 4_000_000 // len(start))
                first = 0
                if bounds is not None:
                    acc += sample(src[:, None])[:, 0]
                    first = 1
                for j0 in range(first, int(J.max()), block):
                    j = torch.arange(j0, min(j0 + block, int(J.max())), device=dev, dtype=F64)
                    p = src[:, None] + (start[:, None] + j * step)[..., None] * n
                    acc += (sample(p) * (j < J[:, None])).sum(1)
                part = torch.zeros_like(tin)
                part[some] = acc
                out[k, r0:r0 + len(yy), x0:x1] += part * 0.15 * 0.25
        if bounds is not None:  # the length of the ray through the pixel's centre
            py, px = torch.meshgrid(yy + 0.5, xx + 0.5, indexing="ij")
            tin, tout = chord(px, py)[1:]
            hits, total = torch.ones_like(tin), torch.clamp(tout - tin, min=0.0)
        length[r0:r0 + len(yy), x0:x1] = torch.where(hits > 0, total / hits, torch.zeros_like(total))
    return (out[0] if bounds is None else out), length


def _taper(w):
    return 1.0 - torch.exp(-9.0 * torch.clamp(w, min=0.0) ** 2)


def _crop_factor(W, H, p, dev):
    """The mask of the volume's shadow with corners p = (A, B, C, D): cut 10, fade over 20 pixels."""
    y, x = torch.meshgrid(torch.arange(H, device=dev, dtype=F64), torch.arange(W, device=dev, dtype=F64), indexing="ij")
    A, B, C, D = [(float(p[2 * i]), float(p[2 * i + 1])) for i in range(4)]

    def side(a, b):  # the half plane of b seen from a
        return (b[0] - a[0]) * (y - a[1]) - (b[1] - a[1]) * (x - a[0])

    def distance(a, b):
        dx, dy = b[0] - a[0], b[1] - a[1]
        l2 = dx * dx + dy * dy
        t = torch.clamp(((x - a[0]) * dx + (y - a[1]) * dy) / l2, 0.0, 1.0) if l2 else torch.zeros_like(x)
        return torch.sqrt((x - a[0] - t * dx) ** 2 + (y - a[1] - t * dy) ** 2)

    inside = (side(A, B) < 0) & (side(D, C) < 0) & (side(C, A) < 0) & (side(B, D) < 0)
    mx = torch.minimum(torch.minimum(distance(A, B), distance(D, C)), torch.minimum(x, W - x - 1))
    my = torch.minimum(torch.minimum(distance(C, A), distance(B, D)), torch.minimum(y, H - y - 1))
    fx = torch.where(mx < 30.0, _taper((mx - 10.0) / 20.0), torch.ones_like(mx))
    fy = torch.where(my < 30.0, _taper((my - 10.0) / 20.0), torch.ones_like(my))
    return torch.where(inside, fx * fy, torch.zeros_like(fx))


def _shadow(f, place):
    """Corners of the volume's shadow in whole pixels, decided in 32 bits."""
    f32 = np.float32
    n, det = f["n"].astype(f32), f["det"].astype(f32)
    frame = np.zeros((4, 4))
    frame[0, :3], frame[1, :3], frame[2, :3], frame[3, :3], frame[3, 3] = f["u"], f["v"], f["n"], f["det"], 1.0
    M = np.linalg.inv(frame).T.astype(f32)
    lo, hi = place["lo"].astype(f32), (place["lo"] + place["size"]).astype(f32)
    P = []
    for c in range(8):
        q = np.array([hi[0] if c & 4 else lo[0], hi[1] if c & 2 else lo[1], hi[2] if c & 1 else lo[2]], f32)
        t = f32(f32(n[0] * q[0] + n[1] * q[1]) + n[2] * q[2])
        t = abs(f32(t + f32(f32(-n[0] * det[0] - n[1] * det[1]) - n[2] * det[2])))
        h = [f32(t * -n[k] + q[k]) for k in range(3)]
        P.append([f32(f32(f32(M[r, 0] * h[0] + M[r, 1] * h[1]) + M[r, 2] * h[2]) + M[r, 3]) for r in range(2)])
    out = []
    for c in range(4):
        for r in range(2):
            a, b = P[2 * c][r], P[2 * c + 1][r]
            out.append(int(a if abs(a) < abs(b) else b))
    return out


def _square(img, N):
    H, W = img.shape[-2:]
    out = torch.zeros(img.shape[:-2] + (N, N), dtype=F64, device=img.device)
    bx, by = (N - W) // 2, (N - H) // 2
    out[..., by:by + H, bx:bx + W] = img
    return out


def _ctf_filter(img, case, defocus, bounds, k, forward):
    """One slab's image through the CTF (forward) or its Wiener correction."""
    H, W = img.shape
    N = max(W, H)
    dev = img.device
    beta = _beta(case)
    y = torch.arange(N, device=dev, dtype=F64)
    y = torch.where(y > N * 0.5, y - N, y)[:, None]
    x = torch.arange(N // 2 + 1, device=dev, dtype=F64)[None]
    d = round((bounds[k] + DISTANCE) * PIXEL_NM * SLAB_NM) / SLAB_NM + SLAB_NM / 2
    d0, d1 = (float(defocus[0]) + d) * 1e-9, (float(defocus[1]) + d) * 1e-9
    volts = 2 * 511 * KV * 1e6 + KV * KV * 1e6
    lam = 6.63e-34 * 3.00e8 / math.sqrt(volts * 1.602e-19 ** 2)
    alpha = torch.where(x == 0, torch.full_like(y * x, math.pi / 2), torch.atan2(y + 0 * x, x + 0 * y))
    z = d0 + (1 - torch.cos(2 * (alpha - math.radians(float(defocus[2]))))) * (d1 - d0)
    radius = torch.sqrt(x * x + y * y)
    q = radius * (1.0 / (PIXEL_NM * 1e-9 * 2)) / (N / 2)
    m = math.pi / 2 * (CS_MM * 1e-3 * lam ** 3 * q ** 4 - 2 * z * lam * q * q)
    l = q / 1e8
    env = torch.exp(-beta[1] * l - beta[2] * l * l - beta[3] * l ** 3)
    if forward:
        val = torch.sin(m) * torch.clamp(env, min=0.01)
        val = torch.where(val.abs() < 1e-4, torch.where(val >= 0, 1e-4, -1e-4).to(F64), val)
        factor = -val
    else:
        val = torch.sin(m) * torch.clamp(env, min=WIENER)
        factor = -val / (val * val + WIENER)
    factor = torch.where(radius > beta[0], factor, torch.ones_like(factor))
    sq = torch.fft.irfft2(torch.fft.rfft2(_square(img, N)) * factor, s=(N, N))
    bx, by = (N - W) // 2, (N - H) // 2
    return sq[by:by + H, bx:bx + W]


def _forward64(vol, f, case, place, whole, mag, defocus, roi=None):
    """ForwardProjection: image and ray lengths, with the CTF slab by slab."""
    W, H = case["W"], case["H"]
    if not case["ctf"]:
        return _project64(vol, f, place, W, H, mag, roi)
    bounds = _slabs(f, whole)
    slabs, length = _project64(vol, f, place, W, H, mag, roi, bounds)
    mask = _crop_factor(W, H, (0, H - 1, W - 1, H - 1, 0, 0, W - 1, 0), vol.device)
    img = sum(mask * _ctf_filter(mask * slabs[k], case, defocus, bounds, k, True) for k in range(len(slabs)))
    return img, length


def _compare64(real, img, length, f, whole):
    """Residual per unit length, faded at the upper detector borders (no crop, fade length 1)."""
    H, W = real.shape
    zmin, zmax = whole["lo"][2], whole["lo"][2] + whole["size"][2]
    thick = abs((DISTANCE - zmin) / f["n"][2] - (DISTANCE - zmax) / f["n"][2])
    res = torch.where(length >= 1.0, (real - img / length * thick) / thick, torch.zeros_like(img))
    y = torch.arange(H, device=real.device, dtype=F64)[:, None]
    x = torch.arange(W, device=real.device, dtype=F64)[None]
    yb = torch.where(y < 1, _taper(y), torch.ones_like(y))
    ya = torch.where(y > H - 2, _taper((H - y - 1) - (H - 1)), torch.ones_like(y))
    xb = torch.where(x < 1, _taper(x), torch.ones_like(x))
    xa = torch.where(x > W - 2, _taper((W - x - 1) - (W - 1)), torch.ones_like(x))
    return xa * xb * ya * yb * res


def _back64(vol, images, f, place, os, inv, weight, bounds=None):
    """vol += weight * sum(sample * chord) / sum(chord) over the sub-pixel samples of each voxel's shadow. Quads of four
    voxels share the samples' bounding rectangle and, with `bounds`, the slab whose image is read (bilinear; nearest
    without)."""
    nx, ny, nz = place["dims"]
    dev = vol.device
    H, W = images.shape[-2:]
    lo = place["lo"]
    n, det, u, v = f["n"], f["det"], f["u"], f["v"]
    U, V = f["to_detector"][0], f["to_detector"][1]
    hu, hv = 0.5 * np.abs(U).sum() * 1.0001 + 1e-5, 0.5 * np.abs(V).sum() * 1.0001 + 1e-5
    nq = 4 * (nx // 4)
    x = torch.arange(nq, device=dev, dtype=F64)[None, None]
    y = torch.arange(ny, device=dev, dtype=F64)[None, :, None]
    planes = max(1, 3_000_000 // (ny * max(nq, 1)))
    for z0 in range(0, nz, planes):
        z = torch.arange(z0, min(z0 + planes, nz), device=dev, dtype=F64)[:, None, None]
        # the quad's rectangle: its 5 x 1 x 1 cell's corners projected, their box's two corners mapped to the detector
        q = 4 * torch.floor(x / 4)
        lower, upper, depth = [None] * 3, [None] * 3, None
        for cx in (0, 5):
            for cy in (0, 1):
                for cz in (0, 1):
                    p = (lo[0] + q + cx + 0 * y + 0 * z, lo[1] + y + cy + 0 * x + 0 * z, lo[2] + z + cz + 0 * x + 0 * y)
                    t = (sum(n[k] * p[k] for k in range(3)) - float(n @ det)).abs()
                    depth = t if depth is None else depth
                    for k in range(3):
                        h = p[k] - t * n[k]
                        lower[k] = h if lower[k] is None else torch.minimum(lower[k], h)
                        upper[k] = h if upper[k] is None else torch.maximum(upper[k], h)
        if n[0] <= 0:
            lower[0], upper[0] = upper[0], lower[0]

        def extent(D, top):
            a = sum(D[k] * (lower[k] - det[k]) for k in range(3))
            b = sum(D[k] * (upper[k] - det[k]) for k in range(3))
            return (torch.clamp(torch.floor(torch.minimum(a, b)), 0, top),
                    torch.clamp(torch.ceil(torch.maximum(a, b)), 0, top))

        ulo, uhi = extent(U, W - 1)
        vlo, vhi = extent(V, H - 1)
        c = (lo[0] + x + 0.5, lo[1] + y + 0.5, lo[2] + z + 0.5)
        uc = sum(U[k] * (c[k] - det[k]) for k in range(3))
        vc = sum(V[k] * (c[k] - det[k]) for k in range(3))
        mu0 = torch.maximum(torch.ceil((uc - hu) * os - 0.5), ulo * os)
        mv0 = torch.maximum(torch.ceil((vc - hv) * os - 0.5), vlo * os)
        num, den = torch.zeros_like(uc), torch.zeros_like(uc)
        if bounds is not None:
            edges = torch.tensor(bounds, device=dev, dtype=F64)
            slab = torch.bucketize(depth.contiguous(), edges, right=True) - 1
            in_slab = (slab >= 0) & (slab < len(bounds) - 1)
            slab = slab.clamp(0, len(bounds) - 2)
        flat = images.reshape(-1)
        for i in range(int(2 * hu * os) + 1):
            pu = (mu0 + i + 0.5) / os
            for j in range(int(2 * hv * os) + 1):
                pv = (mv0 + j + 0.5) / os
                tin, tout = torch.full_like(uc, -1e30), torch.full_like(uc, 1e30)
                for k in range(3):
                    d = (pu - uc) * u[k] + (pv - vc) * v[k]
                    if abs(n[k]) <= 1e-6:  # the ray runs along these faces
                        tout = torch.where(d.abs() < 0.5, tout, torch.full_like(tout, -2e30))
                    else:
                        near, far = (-0.5, 0.5) if n[k] > 0 else (0.5, -0.5)
                        tin = torch.maximum(tin, (near - d) / n[k])
                        tout = torch.minimum(tout, (far - d) / n[k])
                chord = torch.clamp(tout - tin, min=0.0) * (pu < uhi) * (pv < vhi)
                su, sv = inv[0] * pu + inv[1] * pv + inv[2], inv[3] * pu + inv[4] * pv + inv[5]
                if bounds is None:
                    ix, iy = torch.floor(su).clamp(0, W - 1).long(), torch.floor(sv).clamp(0, H - 1).long()
                    val = flat[iy * W + ix]
                else:
                    fx, fy = torch.floor(su - 0.5), torch.floor(sv - 0.5)
                    a, b = su - 0.5 - fx, sv - 0.5 - fy
                    xa, xb = fx.clamp(0, W - 1).long(), (fx + 1).clamp(0, W - 1).long()
                    ya, yb = fy.clamp(0, H - 1).long(), (fy + 1).clamp(0, H - 1).long()
                    base = slab * (H * W)
                    val = (1 - b) * ((1 - a) * flat[base + ya * W + xa] + a * flat[base + ya * W + xb]) + \
                        b * ((1 - a) * flat[base + yb * W + xa] + a * flat[base + yb * W + xb])
                num += val * chord
                den += chord
        good = den > 0
        if bounds is not None:
            good = good & in_slab
        z1 = min(z0 + planes, nz)
        vol[z0:z1, :, :nq] += torch.where(good, weight * num / torch.where(good, den, torch.ones_like(den)),
                                          torch.zeros_like(den))


IDENTITY = np.eye(3).ravel()


def _sart64(case, seed):
    gen = _generator(seed)
    place = _place((case["nx"], case["ny"], case["nz"]))
    vol = _density((case["nz"], case["ny"], case["nx"]), gen).to(DTYPES[case["dtype"]]).to(F64)
    real = _images(case, gen, case["n"]).to(F64)
    frames, defocus = _frames(case, seed), _alignment(case, seed)[4]
    mag, inv = (np.asarray(a, np.float64) if a is not None else IDENTITY for a in _matrices64(case))
    order, W, H = _order(case, seed), case["W"], case["H"]
    for s0 in range(0, case["n"], case["sirt"]):
        subset = [int(i) for i in order[s0:s0 + case["sirt"]]]
        residuals = []
        for i in subset:
            img, length = _forward64(vol, frames[i], case, place, place, mag, defocus[i])
            residuals.append(_compare64(real[i], img, length, frames[i], place))
        for i, res in zip(subset, residuals):
            mask = _crop_factor(W, H, _shadow(frames[i], place), vol.device)
            if case["ctf"]:
                bounds = _slabs(frames[i], place)
                slabs = torch.stack([mask * _ctf_filter(mask ** (k + 1) * res, case, defocus[i], bounds, k, False)
                                     for k in range(len(bounds) - 1)])
                _back64(vol, slabs, frames[i], place, case["os"], inv, 0.5 / case["sirt"], bounds)
            else:
                _back64(vol, (mask * res)[None], frames[i], place, case["os"], inv, 0.5 / case["sirt"])
    return vol


def _matrices64(case):
    """The anisotropy matrix and its inverse: stretch by `aniso` along 35 degrees about the detector's centre."""
    if case["aniso"] == 1.0:
        return None, None
    out = []
    for amount in (case["aniso"], 1.0 / case["aniso"]):
        centre = np.array([[1, 0, case["W"] / 2], [0, 1, case["H"] / 2], [0, 0, 1.0]])
        back = np.array([[1, 0, -case["W"] / 2], [0, 1, -case["H"] / 2], [0, 0, 1.0]])
        out.append((centre @ _rotation("z", -35.0) @ np.diag([amount, 1, 1]) @ _rotation("z", 35.0) @ back).ravel())
    return out


def _subvol64(case, seed):
    gen = _generator(seed)
    whole = _place((case["nx"], case["ny"], case["nz"]))
    sizes, pos, extra = _particles(case, seed)
    real, defocus = _images(case, gen, case["n"]).to(F64), _alignment(case, seed)[4]
    boxes = [torch.zeros((int(z),) * 3, dtype=F64, device=_device()) for z in sizes]
    places = [_place((z, z, z), -0.5 * z + p.astype(np.float64) - 1 + whole["lo"]) for z, p in zip(sizes, pos)]
    frames = [_frames(case, seed, extra[p]) for p in range(len(sizes))]
    plain = _frames(case, seed)
    for i in range(case["n"]):
        bounds = None
        images = real[i][None]
        if case["ctf"]:
            bounds = _slabs(plain[i], whole)
            images = torch.stack([_ctf_filter(real[i], case, defocus[i], bounds, k, False)
                                  for k in range(len(bounds) - 1)])
        for p, box in enumerate(boxes):
            _back64(box, images, frames[p][i], places[p], case["os"], IDENTITY, 1.0, bounds)
    return torch.cat([b.view(-1) for b in boxes])


def _loss64(case, seed):
    """Loss, its gradients and the Gauss-Newton terms of every tilt, and the sum of the volume gradients: the rays keep
    their unshifted sample sets, every sample moves by the shift along the pixel axes."""
    gen = _generator(seed)
    dims = (case["nx"], case["ny"], case["nz"])
    place = _place(dims)
    vol = _density(dims[::-1], gen).to(F64)
    real = _images(case, gen, case["n"], noise=5.0).to(F64)
    shifts = np.random.default_rng(int(seed) + 2).uniform(-1.0, 1.0, (case["n"], 2)).astype(np.float32)
    dev = vol.device
    sums = torch.zeros((case["n"], 6), dtype=F64, device=dev)
    grad = torch.zeros(vol.numel(), dtype=F64, device=dev)
    lo, size = torch.tensor(place["lo"], device=dev), torch.tensor(place["size"], device=dev)
    top = torch.tensor([d - 1 for d in dims], device=dev)
    strides = torch.tensor([1, dims[0], dims[0] * dims[1]], device=dev)
    flat, step, kappa = vol.reshape(-1), round(0.15 * 1024) / 1024, 0.15 * 0.25
    W, H = case["W"], case["H"]

    def corners(p):
        q = p - lo - 0.5
        base = torch.floor(q)
        w, base = q - base, base.long()
        for k in range(8):
            bits = torch.tensor([k & 1, k >> 1 & 1, k >> 2], device=dev)
            index = (torch.minimum(torch.clamp(base + bits, min=0), top) * strides).sum(-1)
            f = torch.where(bits > 0, w, 1 - w)
            sign = 2.0 * bits - 1.0
            yield index, f, sign

    for i, f in enumerate(_frames(case, seed)):
        det, u, v, n = (torch.tensor(f[k], device=dev) for k in ("det", "u", "v", "n"))
        move = float(shifts[i, 0]) * u + float(shifts[i, 1]) * v
        rows = max(1, 4000 // W)
        for r0 in range(0, H, rows):
            yy = torch.arange(r0, min(r0 + rows, H), device=dev, dtype=F64)
            xx = torch.arange(W, device=dev, dtype=F64)
            got, rays = torch.zeros((3, len(yy), W), dtype=F64, device=dev), []
            for ox, oy in ((0.25, 0.25), (0.25, 0.75), (0.75, 0.25), (0.75, 0.75)):
                py, px = torch.meshgrid(yy + oy, xx + ox, indexing="ij")
                s = det + px[..., None] * u + py[..., None] * v
                a, b = torch.nan_to_num((lo - s) / n, nan=-1e30), torch.nan_to_num((lo + size - s) / n, nan=1e30)
                tin, tout = torch.minimum(a, b).amax(-1), torch.maximum(a, b).amin(-1)
                J = torch.where(tout > tin, torch.floor((tout - tin) / step) + 1, torch.zeros_like(tin))
                block = max(1, 1_000_000 // J.numel())
                for j0 in range(0, int(J.max()), block):
                    j = torch.arange(j0, min(j0 + block, int(J.max())), device=dev, dtype=F64)
                    p = s[..., None, :] + (tin[..., None] + j * step)[..., None] * n + move
                    rays.append((p, (j < J[..., None]).to(F64)))
                    for index, w, sign in corners(p):
                        val = flat[index] * rays[-1][1]
                        got[0] += (val * w.prod(-1)).sum(-1)
                        g = torch.stack([sign[0] * w[..., 1] * w[..., 2], sign[1] * w[..., 0] * w[..., 2],
                                         sign[2] * w[..., 0] * w[..., 1]], -1)
                        got[1] += (val * (g @ u)).sum(-1)
                        got[2] += (val * (g @ v)).sum(-1)
            got *= kappa
            r = got[0] - real[i, r0:r0 + len(yy)]
            sums[i] += torch.stack([0.5 * (r * r).sum(), (r * got[1]).sum(), (r * got[2]).sum(), (got[1] ** 2).sum(),
                                    (got[1] * got[2]).sum(), (got[2] ** 2).sum()])
            for p, there in rays:
                for index, w, _ in corners(p):
                    grad.index_add_(0, index.reshape(-1), (w.prod(-1) * there * (r * kappa)[..., None]).reshape(-1))
    return dict(sums=sums, grad=grad.view(vol.shape))


def _refine64(case, seed):
    gen = _generator(seed)
    dims, box = (case["nx"], case["ny"], case["nz"]), case["box"]
    whole = _place(dims)
    vol = _density(dims[::-1], gen).to(F64)
    real = _images(case, gen, case["n"]).to(F64)
    model = _density((box,) * 3, gen).to(F64)
    pos, angles, rois = _refinement(case, seed)
    place = _place((box,) * 3, -0.5 * box + pos.astype(np.float64) - 1 + whole["lo"])
    # the model turned about its voxel box // 2: out(p) = in(c + R^T (p - c))
    R = _rotation("z", angles[1]) @ _rotation("x", angles[2]) @ _rotation("z", angles[0])
    R = torch.tensor(R, device=_device())
    r = torch.arange(box, device=_device(), dtype=F64) - box // 2
    z, y, x = torch.meshgrid(r, r, r, indexing="ij")
    q = torch.clamp(torch.stack([x, y, z], -1) @ R + box // 2, 0, box - 1)
    model = torch.nn.functional.grid_sample(model[None, None], (2 * q / (box - 1) - 1)[None], mode="bilinear",
                                            padding_mode="border", align_corners=True)[0, 0]
    frames, defocus = _frames(case, seed), _alignment(case, seed)[4]
    W, H = case["W"], case["H"]
    N = max(W, H)
    bx, by = (N - W) // 2, (N - H) // 2
    ix, iy = (torch.arange(N, device=_device()) - b for b in (bx, by))
    ix, iy = (torch.where(i < 0, -i - 1, torch.where(i >= m, 2 * m - i - 1, i)) for i, m in ((ix, W), (iy, H)))
    residual, maps, found, peaks = [], [], [], []
    for i, f in enumerate(frames):
        img, length = _forward64(vol, f, case, whole, whole, IDENTITY, defocus[i], rois[i])
        residual.append(_compare64(real[i], img, length, f, whole))
        # the box's slabs are cut on the box
        img, _ = _forward64(model, f, case, place, place, IDENTITY, defocus[i], rois[i])
        a, b = (t[iy][:, ix] - t[iy][:, ix].mean() for t in (residual[-1], img))
        cc = torch.fft.irfft2(torch.fft.rfft2(a).conj() * torch.fft.rfft2(b), s=(N, N)) / torch.sqrt((a * a).sum() *
                                                                                                   (b * b).sum())
        maps.append(torch.roll(cc, (20, 20), (0, 1))[:40, :40])
        k = torch.arange(N, device=_device(), dtype=F64)
        k = torch.where(k > N // 2, k - N, k)
        cc = torch.where(k[:, None] ** 2 + k[None] ** 2 > 100.0, torch.zeros_like(cc), cc)
        at = int(cc.argmax())
        peaks.append(float(cc.view(-1)[at]))
        found.append([int(k[at % N]), int(k[at // N])])
    return dict(residual=torch.stack(residual), maps=torch.stack(maps), shifts=None, peaks=np.array(peaks))


def _prepare64(case, seed):
    raw = _raw_frames(case, _generator(seed))
    W, H = case["W"], case["H"]
    N = max(W, H)
    bx, by = (N - W) // 2, (N - H) // 2
    dev = _device()
    ix, iy = (torch.arange(N, device=dev) - b for b in (bx, by))
    ix, iy = (torch.where(i < 0, -i - 1, torch.where(i >= m, 2 * m - i - 1, i)) for i, m in ((ix, W), (iy, H)))
    x = torch.arange(N // 2 + 1, device=dev, dtype=F64)[None]
    y = torch.arange(N, device=dev, dtype=F64)
    y = torch.where(y > N * 0.5, y - N, y)[:, None]
    dist = torch.sqrt(x * x + y * y)
    lp, hp, lps, hps = FILTER["lp"] - FILTER["lps"], FILTER["hp"] + FILTER["hps"], FILTER["lps"], FILTER["hps"]
    fil = (dist <= lp).to(F64)
    soft = (1 - fil) * torch.exp(-(dist - lp) ** 2 / (2 * lps * lps))
    fil = torch.where(soft > 0.001, soft, fil)
    high = (dist >= hp).to(F64)
    fil = fil * high
    soft = (1 - high) * torch.exp(-(dist - hp) ** 2 / (2 * hps * hps))
    fil = torch.where(soft > 0.001, soft, fil)
    images, stats = [], []
    for i in range(case["n"]):
        img = (raw[i].view(torch.int16) if case["raw"] == "uint16" else raw[i]).to(F64)
        sq = img[iy][:, ix]
        mean = sq.mean()
        sq = torch.where(sq > FILTER["bad_pixel_value"] * mean, mean, sq)
        out = torch.fft.irfft2(torch.fft.rfft2(sq) * fil, s=(N, N))[by:by + H, bx:bx + W]
        mean, std = out.mean(), out.std(unbiased=False)
        images.append((out - mean) / -std)
        stats.append([float(mean), float(std)])
    return dict(images=torch.stack(images), stats=None, bad=None)


def exact(case, seed):
    op = case["op"]
    if op == "prepare":
        return _prepare64(case, seed)
    samples = case["n"] * 4.0 * case["W"] * case["H"] * case["nz"] * 1.4 / 0.15
    if op in ("sart", "project", "refine") and samples > 2.1e10:
        return None
    if op == "loss" and samples > 4e9:
        return None
    if op == "sart":
        return _sart64(case, seed)
    if op == "project":
        gen = _generator(seed)
        place = _place((case["nx"], case["ny"], case["nz"]))
        vol = _density((case["nz"], case["ny"], case["nx"]), gen).to(DTYPES[case["dtype"]]).to(F64)
        mag = _matrices64(case)[0]
        mag = IDENTITY if mag is None else mag
        got = [_forward64(vol, f, case, place, place, mag, d)
               for f, d in zip(_frames(case, seed), _alignment(case, seed)[4])]
        return torch.stack([torch.stack([g[k] for g in got]) for k in (0, 1)])
    if op == "subvol":
        return _subvol64(case, seed) if case["particles"] * case["n"] <= 3000 else None
    if op == "loss":
        return _loss64(case, seed)
    return _refine64(case, seed)
