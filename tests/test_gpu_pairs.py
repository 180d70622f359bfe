"""The packed pair kernels (the default path of every convolution) at the edges of their shapes.

Each case is one convolution through the C ABI against the FP64 oracle, with the tolerance of the
other convolution tests (FP32 transforms: max abs error <= 2e-6 of the output's maximum).  The
sizes reach single slices and rows, lengths of one to three z stages, several tiles per axis with
clipped last ones, planes that leave one CTA per SM, rows whose length and start allow 16-, 8- or
only 4-byte accesses, and kernels wider than the volume (more than one reflection)."""
import numpy as np
import pytest

from oracle import mvdecon_oracle as O
from spim_registration_gb300 import FLAG_AUTOTUNE, Deconvolution, native
from spim_registration_gb300 import synthetic as S
from tests.helpers import rel_l2, rel_max

pytestmark = pytest.mark.gpu

TOL = 2e-6


@pytest.mark.parametrize("shape,kshape", [
    ((1, 1, 1), (1, 1, 1)),
    ((1, 1, 5), (1, 1, 1)),
    ((1, 7, 6), (1, 5, 3)),
    ((2, 3, 4), (7, 9, 11)),            # kernel several times the volume
    ((13, 17, 19), (3, 5, 7)),
    ((40, 33, 34), (9, 15, 15)),        # odd rows; x starts that are not even
    ((90, 41, 60), (11, 7, 9)),         # three z stages
    ((33, 70, 130), (9, 21, 31)),       # several tiles in y, clipped last ones
    ((20, 260, 300), (5, 31, 33)),      # planes beyond half an SM's shared memory
    ((410, 24, 20), (31, 3, 3)),        # several tiles along z
    ((12, 50, 515), (3, 3, 65)),        # several tiles along x, odd rows
])
@pytest.mark.parametrize("mode,value", [(O.MIRROR, 0.0), (O.VALUE, 1.0)])
def test_device_convolution_matches_fp64(shape, kshape, mode, value):
    torch = pytest.importorskip("torch")
    lib = native.load()
    rng = np.random.default_rng(sum(shape) + sum(kshape))
    x = (rng.random(shape) * 100).astype(np.float32)
    k = rng.random(kshape).astype(np.float32)
    k /= k.sum()
    xd, kd = torch.from_numpy(x).cuda(), torch.from_numpy(k).cuda()
    out = torch.full_like(xd, float("nan"))
    torch.cuda.synchronize()
    native.check(lib.mvd_convolve3d_device(xd.data_ptr(), out.data_ptr(), native.iarr(shape[::-1]), kd.data_ptr(),
                                           native.iarr(kshape[::-1]), 0 if mode == O.MIRROR else 1, value, 0, None))
    got = out.cpu().numpy()
    assert np.isfinite(got).all()
    assert rel_max(got, O.conv_extended(x, k, mode, value)) < TOL


@pytest.mark.parametrize("nz,kz", [(5, 3), (20, 5), (60, 13), (78, 13), (108, 13), (120, 31), (136, 15), (212, 29),
                                   (224, 31), (260, 61)])
def test_z_lengths_match_fp64(nz, kz):
    """The z pass at lengths of every CTA size (64, 128 and 160 threads) and their remainders, with
    planes that end in the middle of a chunk of pencil pairs."""
    torch = pytest.importorskip("torch")
    lib = native.load()
    rng = np.random.default_rng(nz)
    shape, kshape = (nz, 70, 76), (kz, 5, 7)
    x = (rng.random(shape) * 100).astype(np.float32)
    k = rng.random(kshape).astype(np.float32)
    k /= k.sum()
    xd, kd = torch.from_numpy(x).cuda(), torch.from_numpy(k).cuda()
    out = torch.full_like(xd, float("nan"))
    torch.cuda.synchronize()
    native.check(lib.mvd_convolve3d_device(xd.data_ptr(), out.data_ptr(), native.iarr(shape[::-1]), kd.data_ptr(),
                                           native.iarr(kshape[::-1]), 0, 0.0, 0, None))
    assert rel_max(out.cpu().numpy(), O.conv_extended(x, k, O.MIRROR, 0.0)) < TOL


@pytest.mark.parametrize("shape,lo,hi", [
    ((61, 53, 47), (0, 0, 0), (61, 53, 47)),
    ((64, 56, 48), (3, 5, 2), (60, 51, 47)),   # data boxes at odd positions, aligned rows
    ((62, 50, 40), (1, 0, 4), (62, 49, 31)),   # rows aligned to 8 bytes only
])
def test_deconvolution_of_boxes_matches_fp64(shape, lo, hi):
    """Views whose data fill a box (x, y, z) of the volume only: value-extended tiles, epilogue rows
    that start anywhere, and the statistics of the update pass."""
    p = S.make_problem(2, shape_xyz=shape, psf_size_xyz=(9, 9, 17), n_blobs=25, iterations=3, n_views=2)
    for a in p.views + p.weights:
        keep = a[lo[2]:hi[2], lo[1]:hi[1], lo[0]:hi[0]].copy()
        a[...] = 0
        a[lo[2]:hi[2], lo[1]:hi[1], lo[0]:hi[0]] = keep
    ref, od = O.deconvolve(p, arith="f64", block=None, mask=False)
    with Deconvolution(p.views, p.weights, p.psfs, p.psftype, p.lam) as d:
        assert all(d.plan(v)["kernels"] == "paired" for v in range(2))
        d.run(p.iterations)
        assert rel_l2(d.get_psi(), ref) < 1e-5
        for v in range(2):
            s, m = d.stats(p.iterations - 1, v)
            _, _, rs, rm = [x for x in od.stats if x[0] == p.iterations - 1 and x[1] == v][0]
            assert s == pytest.approx(rs, rel=1e-3)
            assert m == pytest.approx(rm, rel=1e-3, abs=1e-6)


@pytest.mark.parametrize("shape,kshape,paired", [
    ((64, 128, 128), (15, 195, 15), False),   # 12 times the padding of the scalar lengths
    ((91, 157, 203), (21, 171, 21), False),   # 2.8 times
    ((91, 157, 203), (21, 141, 21), True),    # 1.9 times
    ((91, 157, 203), (381, 21, 21), False),
    ((91, 157, 203), (21, 21, 481), False),
    ((1, 64, 64), (1, 31, 31), True),         # fewer planes than SMs: any padding
])
def test_kernels_near_the_longest_lengths_take_the_cheaper_plan(shape, kshape, paired):
    """Kernels so long that a pair plan's tiles would be mostly halo run the scalar kernels, whose
    lengths reach further, and either way the convolution is the oracle's."""
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(kshape[1])
    x = (rng.random(shape) * 100 + 1).astype(np.float32)
    k = rng.random(kshape).astype(np.float32)
    k /= k.sum()
    for flags in (0, FLAG_AUTOTUNE):
        with Deconvolution([x], [np.ones(shape, np.float32)], [k], S.INDEPENDENT, 0.0, 0, flags) as d:
            plan = d.plan(0)
        assert (plan["kernels"] == "paired") == paired, plan
    xd, kd = torch.from_numpy(x).cuda(), torch.from_numpy(k).cuda()
    out = torch.full_like(xd, float("nan"))
    torch.cuda.synchronize()
    native.check(native.load().mvd_convolve3d_device(xd.data_ptr(), out.data_ptr(), native.iarr(shape[::-1]),
                                                     kd.data_ptr(), native.iarr(kshape[::-1]), 0, 0.0, 0, None))
    assert rel_max(out.cpu().numpy(), O.conv_extended(x, k, O.MIRROR, 0.0)) < TOL
