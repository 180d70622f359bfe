"""PSF pipeline on the GPU against the oracle: extraction from bead neighbourhoods (periodic
trilinear, summed over the locations), normalisation, the transform into the fused frame and
ExtractPSF's per-view bookkeeping.  FP32 interpolation: max abs error <= 1e-5 of the output's
max."""
import ctypes
import math

import numpy as np
import pytest

from oracle import mvdecon_oracle as O
from spim_registration_gb300 import ExtractPSF, native
from spim_registration_gb300.psf import extract_psf_local, transform_psf

pytestmark = pytest.mark.gpu


def _rot_y(deg, scale=(1.0, 1.0, 1.0), shift=(0.0, 0.0, 0.0)):
    t = math.radians(deg)
    r = np.array([[math.cos(t), 0, math.sin(t)], [0, 1, 0], [-math.sin(t), 0, math.cos(t)]]) @ np.diag(scale)
    return np.concatenate([r, np.asarray(shift, dtype=np.float64)[:, None]], axis=1).ravel()


def _close(got, want, tol=1e-5):
    err = np.abs(got.astype(np.float64) - want).max() / max(np.abs(want).max(), 1e-30)
    assert err <= tol, err


def _beads(rng, shape_zyx, n):
    img = (rng.random(shape_zyx) * 5).astype(np.float32)
    locs = []
    for _ in range(n):
        c = [rng.uniform(0, s) for s in shape_zyx[::-1]]  # anywhere: boxes wrap at the border
        locs.append(c)
        z, y, x = np.meshgrid(*[np.arange(s) for s in shape_zyx], indexing="ij")
        img += (300 * np.exp(-((x - c[0]) ** 2 + (y - c[1]) ** 2) / 2.0 - (z - c[2]) ** 2 / 8.0)).astype(np.float32)
    return img, locs


@pytest.mark.parametrize("normalize", [False, True])
def test_extraction_matches_oracle(normalize):
    rng = np.random.default_rng(11)
    img, locs = _beads(rng, (40, 48, 56), 25)
    got = extract_psf_local(img, locs, (9, 11, 13), normalize=normalize)
    want = O.extract_psf_local(img, locs, (9, 11, 13), normalize=normalize)
    assert got.shape == (13, 11, 9)
    _close(got, want)


@pytest.mark.parametrize("deg,scale", [(0, (1, 1, 1)), (30, (1, 1, 2.5)), (90, (1, 1, 1.7)), (137, (1.2, 0.9, 2))])
def test_transform_matches_oracle(deg, scale):
    rng = np.random.default_rng(deg)
    psf = rng.random((21, 11, 9)).astype(np.float32)
    m = _rot_y(deg, scale, (3.0, -2.0, 7.5))
    got = transform_psf(psf, m)
    dims, off = O.transformed_psf_size((9, 11, 21), m)
    want = O.transform_psf(psf, m, dims, off)
    assert got.shape == tuple(dims[::-1])
    _close(got, want)


def test_extract_psf_class_per_view_and_average():
    rng = np.random.default_rng(12)
    img, locs = _beads(rng, (32, 36, 40), 12)
    ex = ExtractPSF()
    models = {"a": _rot_y(0), "b": _rot_y(45, (1, 1, 2)), "c": _rot_y(90, (1, 1, 1.5))}
    for v, m in models.items():
        ex.extractNextImg(img, v, m, locs, (7, 7, 11))
    assert ex.getViewIdsForPSFs() == list(models)
    want_orig = O.extract_psf_local(img, locs, (7, 7, 11), normalize=True)
    for v, m in models.items():
        _close(ex.getInputCalibrationPSFs()[v], want_orig)
        dims, off = O.transformed_psf_size((7, 7, 11), m)
        _close(ex.getTransformedPSF(v), O.transform_psf(want_orig, m, dims, off))
    avg = ex.computeAverageTransformedPSF()
    assert avg.shape == tuple(ex.computeMaxDimTransformedPSF()[::-1])
    assert avg.sum() == pytest.approx(sum(p.sum() for p in ex.getPSFMap().values()), rel=1e-5)


@pytest.mark.parametrize("shape,psf,beads", [((5, 6, 7), (9, 11, 13), 3),      # PSF larger than the view
                                             ((20, 30, 70), (33, 5, 9), 40),   # partial runs along x, y and z
                                             ((16, 16, 16), (1, 1, 1), 200), ((24, 40, 40), (31, 31, 61), 1)])
def test_extraction_runs_and_bead_chunks_match_oracle(shape, psf, beads):
    """Runs of 4 x 8 voxels and 32 lanes that end inside the PSF, bead counts around the chunk size,
    locations outside the view on both sides (periodic) and on voxel centres."""
    rng = np.random.default_rng(beads)
    img = (rng.random(shape) * 100).astype(np.float32)
    locs = rng.uniform(-2, 3, (beads, 3)) * np.array(shape[::-1])
    locs[0] = np.round(locs[0])
    _close(extract_psf_local(img, locs, psf), O.extract_psf_local(img, locs, psf))


def _extract_on(lib, torch, img, locs_ptr, n, psf, out, stream):
    native.check(lib.mvd_extract_psf(img.data_ptr(), native.iarr(img.shape[::-1]),
                                     ctypes.cast(locs_ptr, ctypes.POINTER(ctypes.c_double)), n, native.iarr(psf),
                                     out.data_ptr(), 0, 0, ctypes.c_void_p(stream.cuda_stream)))


def test_captured_extraction_replays_from_the_callers_locations():
    """A graph captured from the call reads the caller's own (page-locked) array at every replay and
    no host memory of the call's."""
    torch = pytest.importorskip("torch")
    lib = native.load()
    rng = np.random.default_rng(21)
    img = (rng.random((30, 32, 34)) * 100).astype(np.float32)
    first, second = (rng.uniform(0, 30, (40, 3)) for _ in range(2))
    d_img, locs = torch.from_numpy(img).cuda(), torch.from_numpy(first.copy()).pin_memory()
    out = torch.empty((11, 7, 9), device="cuda")
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    _extract_on(lib, torch, d_img, locs.data_ptr(), 40, (9, 7, 11), out, s)
    s.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=s):
        _extract_on(lib, torch, d_img, locs.data_ptr(), 40, (9, 7, 11), out, s)
    for want in (first, second):
        locs.copy_(torch.from_numpy(want))
        out.fill_(float("nan"))
        graph.replay()
        torch.cuda.synchronize()
        _close(out.cpu().numpy(), O.extract_psf_local(img, want, (9, 7, 11)))


def test_extraction_is_done_with_pageable_locations_on_return():
    """The array may be reused as soon as the call returns, with the stream still busy."""
    torch = pytest.importorskip("torch")
    lib = native.load()
    rng = np.random.default_rng(22)
    d_img = torch.from_numpy((rng.random((30, 32, 34)) * 100).astype(np.float32)).cuda()
    locs = rng.uniform(0, 30, (200000, 3))
    outs = [torch.empty((3, 3, 3), device="cuda") for _ in range(2)]
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    for out, busy in zip(outs, (0, 20_000_000)):
        mine = locs.copy()
        with torch.cuda.stream(s):
            torch.cuda._sleep(busy)
        _extract_on(lib, torch, d_img, mine.ctypes.data, len(mine), (3, 3, 3), out, s)
        mine[...] = np.nan
    torch.cuda.synchronize()
    assert torch.equal(outs[0], outs[1]) and torch.isfinite(outs[0]).all()


def test_extraction_of_a_thin_psf_of_many_voxels():
    """A PSF whose runs of 32 lanes hold more threads than an int counts: one voxel per lane's row, each the
    periodic view's own value (a bead on a voxel centre)."""
    torch = pytest.importorskip("torch")
    n = 1 << 28
    img = torch.arange(1, 31, dtype=torch.float32, device="cuda").view(1, 30, 1)
    locs = np.array([[0.0, 11.0, 0.0]])
    out = torch.empty((1, n, 1), device="cuda")
    s = torch.cuda.current_stream()
    _extract_on(native.load(), torch, img, locs.ctypes.data, 1, (1, n, 1), out, s)
    y = (torch.arange(n, device="cuda") - n // 2 + 11) % 30
    assert torch.equal(out.view(-1), (y + 1).float())


def test_extraction_at_the_end_of_an_axis_near_2_to_the_31():
    """Positions in the PSF pass 2^31 before they wrap to the view's start."""
    torch = pytest.importorskip("torch")
    nx = 2**31 - 5
    if torch.cuda.mem_get_info()[0] < 12 * 2**30:
        pytest.skip("needs 9 GB")
    img = torch.zeros((1, 1, nx), device="cuda")
    img[0, 0, -20:] = torch.arange(1, 21, device="cuda")
    img[0, 0, :20] = torch.arange(101, 121, device="cuda")
    locs = np.array([[float(nx - 2), 0.0, 0.0]])
    out = torch.empty((1, 1, 17), device="cuda")
    _extract_on(native.load(), torch, img, locs.ctypes.data, 1, (17, 1, 1), out, torch.cuda.current_stream())
    want = list(range(11, 21)) + list(range(101, 108))  # positions nx - 10 .. nx + 6
    assert out.view(-1).tolist() == want


@pytest.mark.parametrize("beads", [160, 161, 512, 513, 1360, 1361])
def test_beads_by_value_and_by_copy_match_oracle(beads):
    """Bead counts on both sides of each size of the parameter block, and of the copy beyond them; the
    array may be reused when the call returns."""
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(beads)
    img = (rng.random((12, 14, 16)) * 100).astype(np.float32)
    locs = rng.uniform(-20, 40, (beads, 3))
    want = O.extract_psf_local(img, locs, (5, 3, 4))
    d_img, out, s = torch.from_numpy(img).cuda(), torch.empty((4, 3, 5), device="cuda"), torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(s):
        torch.cuda._sleep(5_000_000)
    _extract_on(native.load(), torch, d_img, locs.ctypes.data, beads, (5, 3, 4), out, s)
    locs[...] = np.nan
    s.synchronize()
    _close(out.cpu().numpy(), want)
