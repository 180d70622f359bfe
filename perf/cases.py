"""The work that users of this library have it do, as measurable cases.

Every case goes through the public entry points: the deconvolution handle (``Deconvolution``), the
JNA drop-in convolution, the device convolution, the input preparation, the separable Gaussians
of the interest-point detection, the forward / backward pair of PSF refinement and the PSF
extraction.  ``listed()`` holds twelve of them, from the smallest call to the 4-view 512x512x256
deconvolution; ``draw(rng)`` gives more of the same ranges.  Sizes are (x, y, z).
"""
from __future__ import annotations

import ctypes
import math
import random

import numpy as np
import torch

from spim_registration_gb300 import inputs, mvdecon, native, psf, separable

DEV = "cuda:0"
MIN_VALUE = float(np.float32(1e-4))
OPTIMIZATION_II, OPTIMIZATION_I, EFFICIENT_BAYESIAN, INDEPENDENT = 0, 1, 2, 3


def listed():
    return [
        # The smallest call: a cropped region of interest, two views.  Launches and latency count.
        dict(name="decon 40x32x24 2 views", kind="decon", nx=40, ny=32, nz=24, views=2, kx=7, ky=7, kz=11, psftype=INDEPENDENT,
             lam=0.006, iterations=10, weights="ones", layout=0),
        # A small two-view acquisition with independent update kernels.
        dict(name="decon 128x128x64 2 views", kind="decon", nx=128, ny=128, nz=64, views=2, kx=9, ky=9, kz=25,
             psftype=INDEPENDENT, lam=0.006, iterations=10, weights="ones", layout=0),
        # The ordinary four-view acquisition: blended weights, efficient Bayesian kernels.
        dict(name="decon 256x256x192 4 views", kind="decon", nx=256, ny=256, nz=192, views=4, kx=15, ky=15, kz=41,
             psftype=EFFICIENT_BAYESIAN, lam=0.006, iterations=20, weights="blend", layout=0),
        # Six views that each cover only a part of the fused box: ragged data boxes of their own size.
        dict(name="decon 256x256x256 6 crops", kind="decon", nx=256, ny=256, nz=256, views=6, kx=15, ky=15, kz=41,
             psftype=EFFICIENT_BAYESIAN, lam=0.006, iterations=20, weights="crop", layout=3),
        # The largest: four views of 512x512x256 with wide PSFs.
        dict(name="decon 512x512x256 4 views", kind="decon", nx=512, ny=512, nz=256, views=4, kx=31, ky=31, kz=61,
             psftype=EFFICIENT_BAYESIAN, lam=0.006, iterations=10, weights="blend", layout=0),
        # A whole job on raw stacks of odd sizes: resample, normalise, prepare kernels, iterate, read psi.
        dict(name="job 203x157x91 3 views", kind="job", nx=203, ny=157, nz=91, views=3, kx=11, ky=11, kz=23,
             psftype=OPTIMIZATION_I, lam=0.0, iterations=10, osem=1),
        # The Java host's own loop: one block in host memory, convolved in place through the JNA entry point.
        dict(name="dropin block 128x128x128", kind="dropin", nx=128, ny=128, nz=128, kx=15, ky=15, kz=41),
        # A device-resident volume of odd sizes, zero outside, with a kernel that is new at each call.
        dict(name="conv 301x211x157 k21x21x33", kind="conv", nx=301, ny=211, nz=157, kx=21, ky=21, kz=33, ext=1),
        # Input preparation of the four-view acquisition: anisotropic raw stacks into the fused box.
        dict(name="inputs 256x256x192 4 views", kind="inputs", nx=256, ny=256, nz=192, views=4, zscale=2.5, osem=2, mode=0),
        # Interest-point detection: the two Gaussians of the difference-of-Gaussian detector.
        dict(name="dog 320x288x190 sigma 1.8", kind="dog", nx=320, ny=288, nz=190, sigma=1.8, oob=2),
        # One step of PSF refinement on bead data: new PSFs installed, the likelihood and its gradients.
        dict(name="gradient 192x192x192 4 views", kind="gradient", nx=192, ny=192, nz=192, views=4, kx=31, ky=31, kz=61),
        # PSF extraction of four bead stacks, normalised and transformed into the fused frame.
        dict(name="psf 31x31x61 500 beads", kind="psf", nx=256, ny=256, nz=128, views=4, kx=31, ky=31, kz=61, beads=500,
             zscale=2.0),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _odd(rng, lo, hi):
    return _log_int(rng, lo, hi) | 1


def draw(rng):
    kind = rng.choice(["decon", "decon", "decon", "decon", "job", "dropin", "conv", "inputs", "dog", "gradient", "psf"])
    if kind == "decon":
        while True:
            c = dict(kind=kind, nx=_log_int(rng, 32, 512), ny=_log_int(rng, 32, 512), nz=_log_int(rng, 20, 256),
                     views=rng.randint(1, 6), kx=_odd(rng, 5, 31), ky=_odd(rng, 5, 31), kz=_odd(rng, 9, 61),
                     psftype=rng.choice([EFFICIENT_BAYESIAN, EFFICIENT_BAYESIAN, OPTIMIZATION_I, OPTIMIZATION_II, INDEPENDENT]),
                     lam=rng.choice([0.006, 0.006, 0.0]), iterations=rng.randint(5, 20),
                     weights=rng.choice(["ones", "blend", "blend", "crop"]), layout=rng.randint(0, 99))
            if c["nx"] * c["ny"] * c["nz"] * c["views"] * c["iterations"] <= 1.2e9:
                return c
    if kind == "job":
        return dict(kind=kind, nx=_log_int(rng, 48, 300), ny=_log_int(rng, 48, 300), nz=_log_int(rng, 32, 160),
                    views=rng.randint(2, 4), kx=_odd(rng, 5, 21), ky=_odd(rng, 5, 21), kz=_odd(rng, 9, 41),
                    psftype=rng.choice([EFFICIENT_BAYESIAN, OPTIMIZATION_I, INDEPENDENT]), lam=rng.choice([0.006, 0.0]),
                    iterations=rng.randint(5, 15), osem=rng.choice([0, 1, 2]))
    if kind == "dropin":
        return dict(kind=kind, nx=_log_int(rng, 48, 256), ny=_log_int(rng, 48, 256), nz=_log_int(rng, 48, 160),
                    kx=_odd(rng, 5, 31), ky=_odd(rng, 5, 31), kz=_odd(rng, 9, 45))
    if kind == "conv":
        return dict(kind=kind, nx=_log_int(rng, 24, 400), ny=_log_int(rng, 24, 400), nz=_log_int(rng, 16, 256),
                    kx=_odd(rng, 5, 41), ky=_odd(rng, 5, 41), kz=_odd(rng, 5, 61), ext=rng.choice([0, 1]))
    if kind == "inputs":
        return dict(kind=kind, nx=_log_int(rng, 48, 400), ny=_log_int(rng, 48, 400), nz=_log_int(rng, 32, 256),
                    views=rng.randint(2, 8), zscale=rng.choice([1.0, 2.0, 2.5, 4.0]), osem=rng.choice([0, 1, 2]),
                    mode=rng.choice([0, 0, 1]))
    if kind == "dog":
        return dict(kind=kind, nx=_log_int(rng, 48, 512), ny=_log_int(rng, 48, 512), nz=_log_int(rng, 24, 256),
                    sigma=round(math.exp(rng.uniform(math.log(0.8), math.log(14.0))), 3), oob=rng.choice([0, 1, 2, 2]))
    if kind == "gradient":
        return dict(kind=kind, nx=_log_int(rng, 48, 200), ny=_log_int(rng, 48, 200), nz=_log_int(rng, 48, 200),
                    views=rng.randint(1, 4), kx=_odd(rng, 9, 31), ky=_odd(rng, 9, 31), kz=_odd(rng, 9, 61))
    return dict(kind=kind, nx=_log_int(rng, 96, 400), ny=_log_int(rng, 96, 400), nz=_log_int(rng, 48, 200),
                views=rng.randint(1, 4), kx=_odd(rng, 9, 31), ky=_odd(rng, 9, 31), kz=_odd(rng, 13, 61),
                beads=_log_int(rng, 20, 800), zscale=rng.choice([1.0, 2.0, 3.0]))


# ------------------------------------------------------------------------------------------
# inputs
# ------------------------------------------------------------------------------------------
def _rot_y(deg):
    t = math.radians(deg)
    return np.array([[math.cos(t), 0.0, math.sin(t)], [0.0, 1.0, 0.0], [-math.sin(t), 0.0, math.cos(t)]])


def _angles(views):
    return [180.0 * v / max(views, 1) for v in range(views)]


def _rotated_psf(size_xyz, deg, widen=1.0):
    """A Gaussian of the given box, rotated about y, in the odd bounding box of the rotated one."""
    r = _rot_y(deg)
    dims = [(int(e + 1e-9) + 1) | 1 for e in np.abs(r) @ (np.asarray(size_xyz, dtype=np.float64) - 1)]
    sigma = widen * np.maximum(0.6, np.asarray(size_xyz, dtype=np.float64) * np.array([1 / 12, 1 / 12, 1 / 8.5]))
    ax = [np.arange(n) - n // 2 for n in dims]
    z, y, x = np.meshgrid(ax[2], ax[1], ax[0], indexing="ij")
    local = np.stack([x, y, z], axis=-1) @ r
    g = np.exp(-0.5 * ((local / sigma) ** 2).sum(-1))
    return (g / g.sum()).astype(np.float32)


def _blobs(shape, count, sigma, rng, background=10.0):
    """Gaussian spots of random height on a constant background (a float32 CUDA volume)."""
    n = int(np.prod(shape))
    at = np.unique(rng.integers(0, n, count))
    vol = torch.zeros(n, device=DEV)
    vol[torch.from_numpy(at).to(DEV)] = torch.from_numpy(rng.uniform(100, 1000, at.size).astype(np.float32)).to(DEV)
    vol = vol.view(shape)
    if sigma > 0:
        f = [torch.fft.fftfreq(s, device=DEV) for s in shape[:2]] + [torch.fft.rfftfreq(shape[2], device=DEV)]
        e = [torch.exp(-2 * math.pi ** 2 * sigma ** 2 * q * q) * sigma * math.sqrt(2 * math.pi) for q in f]
        s = torch.fft.rfftn(vol)
        s *= e[0][:, None, None] * e[1][None, :, None]
        s *= e[2][None, None, :]
        vol = torch.fft.irfftn(s, s=shape).clamp_(min=0)
    return vol + background


def _blur(vol, kernel):
    """Periodic blur, for making views only."""
    k = torch.zeros_like(vol)
    kz, ky, kx = [min(a, b) for a, b in zip(kernel.shape, vol.shape)]
    kz, ky, kx = [s if s & 1 else s - 1 for s in (kz, ky, kx)]
    o = [(a - b) // 2 for a, b in zip(kernel.shape, (kz, ky, kx))]
    k[:kz, :ky, :kx] = torch.from_numpy(kernel[o[0]:o[0] + kz, o[1]:o[1] + ky, o[2]:o[2] + kx].copy()).to(DEV)
    k = torch.roll(k, (-(kz // 2), -(ky // 2), -(kx // 2)), (0, 1, 2))
    return torch.fft.irfftn(torch.fft.rfftn(vol) * torch.fft.rfftn(k), s=vol.shape).clamp_(min=0)


def _poisson(vol, seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    return torch.poisson(vol, generator=g)


def _cosine_weight(shape, deg):
    nz, ny, nx = shape
    c = [(n - 1) / 2.0 for n in (nx, ny, nz)]
    z, y, x = [torch.arange(n, device=DEV, dtype=torch.float32) for n in shape]
    z, y, x = z[:, None, None] - c[2], y[None, :, None] - c[1], x[None, None, :] - c[0]
    r = _rot_y(deg)
    w = torch.ones(shape, device=DEV)
    for q, n in (((x * r[0, 0] + z * r[2, 0]) + c[0], nx), (y + c[1], ny), ((x * r[0, 2] + z * r[2, 2]) + c[2], nz)):
        d = torch.minimum(q + 8.0, (n - 1) - q + 8.0).clamp_(0.0, 12.0)
        w = w * (0.5 - 0.5 * torch.cos(math.pi / 12.0 * d))
    return w


def _crop_boxes(case):
    r = random.Random(7000 + case["layout"])
    boxes = []
    for _ in range(case["views"]):
        box = []
        for n in (case["nz"], case["ny"], case["nx"]):
            side = max(1, min(n, int(n * r.uniform(0.375, 1.0))))
            lo = r.randint(0, n - side)
            box.append(slice(lo, lo + side))
        boxes.append(tuple(box))
    return boxes


def _decon_inputs(case, seed):
    shape = (case["nz"], case["ny"], case["nx"])
    rng = np.random.default_rng(seed)
    truth = _blobs(shape, max(8, int(np.prod(shape)) // 40000), 2.0, rng)
    angles = _angles(case["views"])
    psfs = [_rotated_psf((case["kx"], case["ky"], case["kz"]), a) for a in angles]
    views = [_poisson(_blur(truth, p), seed + 101 * (v + 1)).clamp_(min=MIN_VALUE) for v, p in enumerate(psfs)]
    if case["weights"] == "ones":
        weights = [torch.ones(shape, device=DEV) for _ in angles]
    else:
        weights = [_cosine_weight(shape, a) for a in angles]
        if case["weights"] == "crop":
            for k, box in enumerate(_crop_boxes(case)):
                for a in (views, weights):
                    kept = torch.zeros_like(a[k])
                    kept[box] = a[k][box]
                    a[k] = kept
        total = sum(weights).clamp_(min=1.0)
        weights = [w / total for w in weights]
    g = torch.Generator(device=DEV)
    g.manual_seed(seed + 1)
    start = truth.mean() * (1 + 0.05 * torch.rand(shape, generator=g, device=DEV))
    return views, weights, psfs, start


def _pinned(t):
    p = torch.empty(t.shape, dtype=torch.float32, pin_memory=True)
    p.copy_(t)
    return p.numpy()


def _raw_views(case, seed):
    """Raw stacks (coarser along z) and their registrations: rotated about y around the box's centre,
    with a fraction of a voxel of shift."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    s = case.get("zscale", 2.0)
    rng = np.random.default_rng(seed)
    centre = np.array([(nx - 1) / 2, (ny - 1) / 2, (nz - 1) / 2])
    stacks, affines = [], []
    for v, a in enumerate(_angles(case["views"])):
        vx, vy, vz = nx - v % 3, ny + v % 2, max(2, int(nz / s) + v % 2)
        shape = (vz, vy, vx)
        stacks.append(_poisson(_blobs(shape, max(8, int(np.prod(shape)) // 20000), 1.5, rng), seed + 101 * (v + 1)))
        m = _rot_y(a) @ np.diag([1.0, 1.0, s])
        t = centre - m @ np.array([(vx - 1) / 2, (vy - 1) / 2, (vz - 1) / 2]) + np.array([0.3, 0.37, 0.11]) * (v + 1)
        affines.append(np.concatenate([m, t[:, None]], axis=1))
    return stacks, affines


BORDER, BLENDING = (0.0, 0.0, 0.0), (12.0, 12.0, 8.0)


def _beads(case, seed):
    rng = np.random.default_rng(seed)
    shape = (case["nz"], case["ny"], case["nx"])
    stacks, locations, models = [], [], []
    for v, a in enumerate(_angles(case["views"])):
        stacks.append(_poisson(_blobs(shape, case["beads"], 1.6, rng, 20.0), seed + 101 * (v + 1)))
        locations.append(rng.uniform(0, 1, (case["beads"], 3)) * (np.array([case["nx"], case["ny"], case["nz"]]) - 1.0))
        m = _rot_y(a) @ np.diag([1.0, 1.0, case["zscale"]])
        models.append(np.concatenate([m, np.array([[3.5], [-2.25], [7.0]])], axis=1).ravel())
    return stacks, locations, models


# ------------------------------------------------------------------------------------------
# prepare and run
# ------------------------------------------------------------------------------------------
def prepare(case, seed):
    kind = case["kind"]
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    if kind == "decon":
        views, weights, psfs, start = _decon_inputs(case, seed)
        handle = mvdecon.Deconvolution(views, weights, psfs, case["psftype"], case["lam"])
        out = torch.empty((nz, ny, nx), dtype=torch.float32, pin_memory=True).numpy()
        return dict(case=case, handle=handle, start=_pinned(start), out=out)
    if kind == "job":
        stacks, affines = _raw_views(case, seed)
        psfs = [_rotated_psf((case["kx"], case["ky"], case["kz"]), a) for a in _angles(case["views"])]
        out = torch.empty((nz, ny, nx), dtype=torch.float32, pin_memory=True).numpy()
        return dict(case=case, stacks=stacks, affines=affines, psfs=psfs, out=out)
    if kind in ("dropin", "conv"):
        rng = np.random.default_rng(seed)
        block = _poisson(_blobs((nz, ny, nx), max(8, nx * ny * nz // 20000), 2.0, rng), seed)
        kernel = _rotated_psf((case["kx"], case["ky"], case["kz"]), 0.0, rng.uniform(0.8, 1.2))
        if kind == "dropin":
            return dict(case=case, cuda=mvdecon.CUDAFourierConvolution(), volume=block.cpu().numpy(),
                        block=np.empty((nz, ny, nx), dtype=np.float32), kernel=kernel)
        return dict(case=case, lib=native.load(), volume=block, out=torch.empty_like(block),
                    kernel=torch.from_numpy(kernel).to(DEV))
    if kind == "inputs":
        stacks, affines = _raw_views(case, seed)
        return dict(case=case, stacks=stacks, affines=affines)
    if kind == "dog":
        rng = np.random.default_rng(seed)
        volume = _poisson(_blobs((nz, ny, nx), max(8, nx * ny * nz // 20000), 1.6, rng), seed)
        return dict(case=case, lib=native.load(), volume=volume, taps=_dog_taps(case),
                    buffers=[torch.empty_like(volume) for _ in range(4)])
    if kind == "gradient":
        rng = np.random.default_rng(seed)
        shape = (nz, ny, nx)
        truth = _blobs(shape, max(8, nx * ny * nz // 14000), 0.7, rng)
        angles = _angles(case["views"])
        size = (case["kx"], case["ky"], case["kz"])
        views = [_poisson(_blur(truth, _rotated_psf(size, a)), seed + 101 * (v + 1)).clamp_(min=MIN_VALUE)
                 for v, a in enumerate(angles)]
        weights = [_cosine_weight(shape, a) for a in angles]
        wide = [_rotated_psf(size, a, rng.uniform(1.1, 1.3)) for a in angles]
        handle = mvdecon.Deconvolution(views, weights, wide, INDEPENDENT, 0.0)
        handle.set_psi(truth.cpu().numpy())
        return dict(case=case, handle=handle, psfs=wide, truth=truth, views=views, weights=weights)
    stacks, locations, models = _beads(case, seed)
    return dict(case=case, stacks=stacks, locations=locations, models=models)


def _dog_taps(case):
    """The two Gaussians of the detector (the second 2^(1/4) wider), as the detection asks for them."""
    return [separable.get_cuda_kernels([case["sigma"] * f] * 3) for f in (1.0, 2.0 ** 0.25)]


def _prepared_inputs(s):
    """Raw stacks to the fused box: images, blending weights, their overlap and normalisation."""
    c = s["case"]
    made = [inputs.transform_input(v, a, (0, 0, 0), (c["nz"], c["ny"], c["nx"]), BORDER, BLENDING)
            for v, a in zip(s["stacks"], s["affines"])]
    norm = inputs.WeightNormalizer([w for _, w in made], inputs.WeightType(c.get("mode", 0)), 32)
    norm.process()
    norm.apply(norm.osem_speedup(c["osem"]))
    return made, norm


def run(s):
    c = s["case"]
    kind = c["kind"]
    if kind == "decon":  # continue from a given estimate: set it, iterate, read the result
        h = s["handle"]
        h.set_psi(s["start"])
        h.run(c["iterations"])
        return h.get_psi(out=s["out"])
    if kind == "job":
        made, _ = _prepared_inputs(s)
        with mvdecon.Deconvolution([m[0] for m in made], [m[1] for m in made], s["psfs"], c["psftype"], c["lam"]) as h:
            h.run(c["iterations"])
            return h.get_psi(masked=True, out=s["out"])
    if kind == "dropin":
        np.copyto(s["block"], s["volume"])  # the host's block copy
        s["cuda"].convolution3DfftCUDAInPlace(s["block"], s["block"].shape, s["kernel"], s["kernel"].shape, 0)
        return s["block"]
    if kind == "conv":
        k = s["kernel"]
        native.check(s["lib"].mvd_convolve3d_device(
            s["volume"].data_ptr(), s["out"].data_ptr(), native.iarr([c["nx"], c["ny"], c["nz"]]), k.data_ptr(),
            native.iarr(list(k.shape[::-1])), c["ext"], 0.0, 0, None))
        return s["out"]
    if kind == "inputs":
        made, norm = _prepared_inputs(s)
        return [[m[0] for m in made], [m[1] for m in made], norm.getMinOverlappingViews(), norm.getAvgOverlappingViews()]
    if kind == "dog":
        out = []
        for taps, image, scratch in zip(s["taps"], s["buffers"][0::2], s["buffers"][1::2]):
            image.copy_(s["volume"])  # the passes work in place
            got = ctypes.c_void_p()
            native.check(s["lib"].mvd_separable_convolve_device(
                image.data_ptr(), scratch.data_ptr(), (native._F * 3)(*[native.fptr(k) for k in taps]),
                native.iarr([len(k) for k in taps]), native.iarr([c["nx"], c["ny"], c["nz"]]), c["oob"], 5.0, 0,
                ctypes.c_void_p(torch.cuda.current_stream().cuda_stream), ctypes.byref(got)))
            out.append(image if got.value == image.data_ptr() else scratch)
        return out
    if kind == "gradient":
        h = s["handle"]
        for v, k in enumerate(s["psfs"]):
            h.set_kernel(v, 1, k)
        nll = h.forward()
        g, gk = h.backward()
        return [nll, g, gk]
    ex = psf.ExtractPSF()
    for v, (img, model, loc) in enumerate(zip(s["stacks"], s["models"], s["locations"])):
        ex.extractNextImg(img, v, model, loc, (c["kx"], c["ky"], c["kz"]))
    return [[ex.getInputCalibrationPSFs()[v] for v in ex.getViewIdsForPSFs()],
            [ex.getTransformedPSF(v) for v in ex.getViewIdsForPSFs()]]


# ------------------------------------------------------------------------------------------
# what a pass cannot do without
# ------------------------------------------------------------------------------------------
def _conv_flops(n, k):
    """Two real transforms over the extended volume, and the product."""
    m = 1
    for a, b in zip(n, k):
        m *= a + b - 1
    return 2 * 2.5 * m * math.log2(max(2, m)) + 3 * m


def work(case):
    kind = case["kind"]
    n3 = (case["nx"], case["ny"], case["nz"])
    n = n3[0] * n3[1] * n3[2]
    k3 = (case.get("kx", 1), case.get("ky", 1), case.get("kz", 1))
    k = k3[0] * k3[1] * k3[2]
    v = case.get("views", 1)
    if kind in ("decon", "job"):
        part = 1.0
        if case.get("weights") == "crop":
            part = sum((b[0].stop - b[0].start) * (b[1].stop - b[1].start) * (b[2].stop - b[2].start)
                       for b in _crop_boxes(case)) / (v * n)
        # per view stage: psi read and written, the image and its weight read; two convolutions
        w = dict(bytes=case["iterations"] * v * n * 16.0 * part, flops=case["iterations"] * v * 2 * _conv_flops(n3, k3) * part)
        if kind == "job":
            w["bytes"] += v * n * 20.0
            w["flops"] += v * n * 60.0
        return w
    if kind in ("dropin", "conv"):
        return dict(bytes=8.0 * n + 4.0 * k, flops=_conv_flops(n3, k3))
    if kind == "inputs":  # the raw stacks read; images and weights written; weights normalised once more
        return dict(bytes=v * n * (4.0 / case["zscale"] + 8.0 + 8.0), flops=v * n * 80.0)
    if kind == "dog":
        taps = sum(len(t[0]) for t in _dog_taps(case))
        return dict(bytes=2 * 8.0 * n, flops=2.0 * 3 * taps * n)
    if kind == "gradient":  # per view: psi, image and weight read; one convolution forward, three for the gradients
        return dict(bytes=v * n * 24.0 + 4.0 * n, flops=v * 4 * _conv_flops(n3, k3))
    return dict(bytes=v * (4.0 * min(n, 8 * k * case["beads"]) + 8.0 * k), flops=v * case["beads"] * k * 32.0)


# ------------------------------------------------------------------------------------------
# the same results in 64 bits, in plain torch
# ------------------------------------------------------------------------------------------
def _fast_len(n):
    while True:
        m = n
        for f in (2, 3, 5, 7):
            while m % f == 0:
                m //= f
        if m == 1:
            return n
        n += 1


def _mirror(i, n):
    if n == 1:
        return np.zeros_like(i)
    m = np.mod(i, 2 * n - 2)
    return np.where(m < n, m, 2 * n - 2 - m)


class _Conv64:
    """Convolution of volumes of one shape with one centred odd kernel, cropped to the volume."""

    def __init__(self, shape, kernel):
        self.n, self.k = shape, tuple(kernel.shape)
        self.len = [_fast_len(a + b - 1) for a, b in zip(self.n, self.k)]
        self.f = torch.fft.rfftn(kernel.to(DEV, torch.float64), s=self.len)

    def __call__(self, vol, value=None):
        """value None: extended by mirroring, else by that value."""
        lo = [k // 2 for k in self.k]
        if value is None:
            for d in range(3):
                i = _mirror(np.arange(-lo[d], self.n[d] + lo[d]), self.n[d])
                vol = vol.index_select(d, torch.from_numpy(i).to(DEV))
        else:
            vol = torch.nn.functional.pad(vol, (lo[2], lo[2], lo[1], lo[1], lo[0], lo[0]), value=float(value))
        full = torch.fft.irfftn(torch.fft.rfftn(vol, s=self.len) * self.f, s=self.len)
        k, n = self.k, self.n
        return full[k[0] - 1:k[0] - 1 + n[0], k[1] - 1:k[1] - 1 + n[1], k[2] - 1:k[2] - 1 + n[2]].contiguous()


def _kernels64(psfs, psftype):
    """The kernels of both convolutions of an update, per view."""
    p = [torch.from_numpy(q).to(DEV, torch.float64) for q in psfs]
    p = [q / q.sum() for q in p]
    flip = lambda q: q.flip(0, 1, 2)  # noqa: E731
    second = []
    for v, q in enumerate(p):
        others = [w for w in range(len(p)) if w != v]
        if len(p) == 1 or psftype == INDEPENDENT:
            second.append(flip(q))
        elif psftype == EFFICIENT_BAYESIAN:
            k = flip(q)
            for w in others:
                k = k * _Conv64(q.shape, flip(p[w]))(_Conv64(q.shape, p[w])(flip(q), 0.0), 0.0)
            second.append(k / k.sum())
        elif psftype == OPTIMIZATION_I:
            k = q
            for w in others:
                k = k * _Conv64(q.shape, flip(p[w]))(q, 0.0)
            second.append(flip(k / k.sum()))
        else:
            k = q ** len(p)
            second.append(flip(k / k.sum()))
    return p, second


def _iterate64(views, weights, psfs, psftype, lam, psi, iterations):
    k1, k2 = _kernels64(psfs, psftype)
    shape = tuple(psi.shape)
    c1, c2 = [_Conv64(shape, k) for k in k1], [_Conv64(shape, k) for k in k2]
    lam = float(np.float32(lam))
    for _ in range(iterations):
        for v, (img, w) in enumerate(zip(views, weights)):
            img = img.double()
            q = torch.where(img > 0, img / c1[v](psi), torch.ones_like(img))
            value = psi * c2[v](q, 1.0)
            new = (torch.sqrt(1.0 + 2.0 * lam * value) - 1.0) / lam if lam > 0 else value
            new = torch.where(value > 0, new, torch.full_like(new, MIN_VALUE))
            new = torch.where(torch.isnan(new), torch.full_like(new, MIN_VALUE), new.clamp(min=MIN_VALUE))
            psi = psi + (new - psi) * w.double()
    return psi


def _trilinear64(img, t, wrap):
    """Values at the positions t = (x, y, z); wrap(i, n) maps an index, None drops what lies outside."""
    n = img.shape[::-1]
    lo = [torch.floor(q) for q in t]
    fr = [q - f for q, f in zip(t, lo)]
    lo = [f.long() for f in lo]
    flat, acc = img.reshape(-1).double(), 0.0
    for c in range(8):
        b = [c & 1, (c >> 1) & 1, (c >> 2) & 1]
        i, w, ok = [], 1.0, True
        for d in range(3):
            q = lo[d] + b[d]
            w = w * (fr[d] if b[d] else 1.0 - fr[d])
            if wrap is None:
                ok = ok & (q >= 0) & (q < n[d])
                q = q.clamp(0, n[d] - 1)
            else:
                q = wrap(q, n[d])
            i.append(q)
        val = flat[(i[2] * n[1] + i[1]) * n[0] + i[0]]
        acc = acc + (w * val if wrap is not None else w * val * ok)
    return acc


def _mirror_t(i, n):
    if n == 1:
        return torch.zeros_like(i)
    m = torch.remainder(i, 2 * n - 2)
    return torch.where(m < n, m, 2 * n - 2 - m)


def _inputs64(case, seed):
    stacks, affines = _raw_views(case, seed)
    shape = (case["nz"], case["ny"], case["nx"])
    z, y, x = [torch.arange(n, device=DEV, dtype=torch.float64) for n in shape]
    z, y, x = z[:, None, None], y[None, :, None], x[None, None, :]
    table = np.zeros(1001)
    d = 0.0
    while d <= 1.0001:
        table[int(math.floor(d * 1000.0 + 0.5))] = (math.cos((1 - d) * math.pi) + 1) / 2
        d += 0.001
    table = torch.from_numpy(table).to(DEV)
    images, weights = [], []
    for img, a in zip(stacks, affines):
        m = np.linalg.inv(a[:, :3])
        o = -m @ a[:, 3]
        t = [(m[r, 0] * x + m[r, 1] * y + m[r, 2] * z + o[r]).expand(shape) for r in range(3)]
        n = img.shape[::-1]
        inside = torch.ones(shape, dtype=torch.bool, device=DEV)
        w = torch.ones(shape, dtype=torch.float64, device=DEV)
        for q, s, b, r in zip(t, n, BORDER, BLENDING):
            inside &= (q >= 0) & (q < s)
            dist = torch.minimum(q - b, s - 1 - q - b).clamp(min=0.0)
            rel = dist / r
            w = w * torch.where(rel < 1, table[torch.floor(rel.clamp(max=1.0) * 1000.0 + 0.5).long()], torch.ones_like(rel))
            w = torch.where(dist == 0, torch.zeros_like(w), w)
        v = _trilinear64(img, t, _mirror_t).clamp(min=MIN_VALUE)
        images.append(torch.where(inside, v, torch.zeros_like(v)))
        weights.append(w)
    count = sum((w > 0).long() for w in weights)
    low = int(count.min())
    n = count.numel()
    size = n // 32
    flat = count.reshape(-1).double()
    avg = sum(float(flat[p * size:(p + 1) * size if p < 31 else n].mean()) for p in range(32)) / 32
    osem = {0: 1.0, 1: float(max(1, low)), 2: max(1.0, avg)}[case["osem"]]
    total = sum(weights)
    if case.get("mode", 0) == 0:
        total = total.clamp(min=1.0)
    weights = [torch.where(torch.isnan(w / total), w / total, (w / total * osem).clamp(max=1.0)) for w in weights]
    return images, weights, low, avg


def _separable64(vol, taps, oob, value):
    for axis, k in ((2, taps[0]), (1, taps[1]), (0, taps[2])):
        r, n = len(k) // 2, vol.shape[axis]
        if oob == 2:
            ext = vol.index_select(axis, torch.arange(-r, n + r, device=DEV).clamp(0, n - 1))
        else:
            pad = [0] * 6
            pad[2 * (2 - axis)] = pad[2 * (2 - axis) + 1] = r
            ext = torch.nn.functional.pad(vol, pad, value=value if oob == 1 else 0.0)
        out = torch.zeros_like(vol)
        for m in range(2 * r + 1):
            out += float(k[2 * r - m]) * ext.narrow(axis, m, n)
        vol = out
    return vol


def _gradient64(case, seed):
    s = prepare(case, seed)
    psi = s["truth"].double()
    shape = tuple(psi.shape)
    nll, g, gk = 0.0, torch.zeros_like(psi), []
    for img, w, q in zip(s["views"], s["weights"], s["psfs"]):
        k = torch.from_numpy(q).to(DEV, torch.float64)
        img, w = img.double(), w.double()
        f = _Conv64(shape, k)(psi)
        nll += float((w * (f - img * torch.log(f)))[img > 0].sum())
        r = torch.where(img > 0, w * (1 - img / f), torch.zeros_like(f))
        h = [a // 2 for a in k.shape]
        big = [n + 2 * a for n, a in zip(shape, h)]
        ln = [_fast_len(n + 2 * (a - 1)) for n, a in zip(shape, k.shape)]
        idx = [torch.from_numpy(_mirror(np.arange(-a, n + a), n)).to(DEV) for n, a in zip(shape, h)]
        fr = torch.fft.rfftn(r, s=ln)
        # every extended position's share, added to the voxel that it mirrors
        e = torch.fft.irfftn(fr * torch.fft.rfftn(k.flip(0, 1, 2), s=ln), s=ln)[:big[0], :big[1], :big[2]]
        for d in range(3):
            t = torch.zeros([shape[i] if i <= d else big[i] for i in range(3)], dtype=torch.float64, device=DEV)
            e = t.index_add_(d, idx[d], e.contiguous())
        g += e
        ext = psi.index_select(0, idx[0]).index_select(1, idx[1]).index_select(2, idx[2])
        c = torch.fft.irfftn(torch.fft.rfftn(ext, s=ln) * fr.conj(), s=ln)
        gk.append(c[:k.shape[0], :k.shape[1], :k.shape[2]].flip(0, 1, 2).contiguous())
    return [nll, g, gk]


def _psf64(case, seed):
    stacks, locations, models = _beads(case, seed)
    size = (case["kx"], case["ky"], case["kz"])
    z, y, x = [torch.arange(n, device=DEV, dtype=torch.float64) - n // 2 for n in size[::-1]]
    z, y, x = z[:, None, None], y[None, :, None], x[None, None, :]
    box = size[::-1]
    extracted, moved = [], []
    for img, loc, model in zip(stacks, locations, models):
        acc = torch.zeros(box, dtype=torch.float64, device=DEV)
        for b in loc:
            acc += _trilinear64(img, [(q + float(o)).expand(box) for q, o in zip((x, y, z), b)], torch.remainder)
        acc = (acc - acc.min()) / (acc.max() - acc.min())
        extracted.append(acc)
        m = model.reshape(3, 4)
        corners = np.array([[(size[d] - 1.0) * ((c >> d) & 1) for d in range(3)] for c in range(8)]) @ m[:, :3].T + m[:, 3]
        dims = [(int(e) + 1) | 1 for e in corners.max(0) - corners.min(0)]
        off = m[:, :3] @ np.array([s // 2 for s in size], dtype=np.float64) + m[:, 3] - np.array([d // 2 for d in dims])
        inv = np.linalg.inv(m[:, :3])
        pz, py, px = [torch.arange(n, device=DEV, dtype=torch.float64) + o - t for n, o, t in zip(dims[::-1], off[::-1], m[::-1, 3])]
        pz, py, px = pz[:, None, None], py[None, :, None], px[None, None, :]
        t = [(inv[r, 0] * px + inv[r, 1] * py + inv[r, 2] * pz).expand(dims[::-1]) for r in range(3)]
        moved.append(_trilinear64(acc, t, None))
    return [extracted, moved]


def exact(case, seed):
    kind = case["kind"]
    if kind == "decon":
        views, weights, psfs, start = _decon_inputs(case, seed)
        return _iterate64(views, weights, psfs, case["psftype"], case["lam"], start.double(), case["iterations"])
    if kind == "job":
        images, weights, _, _ = _inputs64(case, seed)
        psfs = [_rotated_psf((case["kx"], case["ky"], case["kz"]), a) for a in _angles(case["views"])]
        total, count = sum(images), sum((i > 0).double() for i in images)
        avg = float((total[count > 0] / count[count > 0]).mean()) if bool((count > 0).any()) else 0.5
        psi = _iterate64(images, weights, psfs, case["psftype"], case["lam"], torch.full_like(total, avg), case["iterations"])
        return torch.where(count > 0, psi, torch.zeros_like(psi))
    if kind in ("dropin", "conv"):
        s = prepare(case, seed)
        vol = torch.as_tensor(s["volume"]).to(DEV, torch.float64)
        k = torch.as_tensor(s["kernel"]).to(DEV, torch.float64)
        mirrored = kind == "dropin" or case["ext"] == 0
        return _Conv64(tuple(vol.shape), k)(vol, None if mirrored else 0.0)
    if kind == "inputs":
        images, weights, _, avg = _inputs64(case, seed)
        return [images, weights, None, avg]
    if kind == "dog":
        s = prepare(case, seed)
        return [_separable64(s["volume"].double(), t, case["oob"], 5.0) for t in s["taps"]]
    if kind == "gradient":
        return _gradient64(case, seed)
    return _psf64(case, seed)
