"""Strip-word path (csrc/strip.cu): integer patterns' Radon means from sums over four-pixel strips, and
the peak kernel that reads them.  Integer ray sums are exact in any order and the convolution keeps
the per-stage multiply-add order, so every field equals the per-stage FP32 method's bit for bit;
normmax, whose mean is reduced in another order, to 1e-6 (a few float32 ulps of a mean over more
than 10^4 values).

The sizes lie at the edges of the kernels' tiles: images that fill a strip phase or leave one to three
columns over, unequal sides, the largest table with four and with two strips a phase, one rho segment
and several, theta counts other than 180, one slab and several, units cut short, and more patterns than
one pass of the workspace holds.
"""
import numpy as np
import pytest

import pyebsdindex_gb300 as pg
from pyebsdindex_gb300 import _lib, synthetic as syn

pytestmark = pytest.mark.gpu

FIELDS = ("max", "maxloc", "avemax", "aveloc", "width", "theta", "rho", "valid")


def plan(h, w, nrho, ntheta=180, frac=0.1, mask=True, nbands=9, sigma=1.0):
    bd = pg.BandDetect(nTheta=ntheta, nRho=nrho, tSigma=sigma, rSigma=sigma, rhoMaskFrac=frac, nBands=nbands)
    bd.band_detect_setup(patDim=(h, w), patternmask=syn.circular_mask(h, w) if mask else None)
    return bd


def check(bd, pats):
    want = bd.find_bands(pats, method="plain")
    got = bd.find_bands(pats, method="fused")
    for f in FIELDS:
        assert got[f].tobytes() == want[f].tobytes(), f
    np.testing.assert_allclose(got["normmax"], want["normmax"], rtol=1e-6)


def patterns(n, h, w, dtype, seed):
    peak = 200.0 if dtype == np.uint8 else 4000.0
    return syn.make_patterns(n, h, w, seed=seed, dtype=dtype, peak=peak, noise_frac=0.2)[0]


@pytest.mark.parametrize("dtype", [np.uint8, np.uint16])
@pytest.mark.parametrize("h,w,nrho,ntheta", [
    (40, 40, 60, 180), (45, 64, 64, 180), (63, 49, 96, 180), (61, 83, 92, 180), (80, 80, 120, 180),
    (84, 84, 126, 180), (80, 80, 119, 90), (60, 60, 90, 97), (101, 120, 151, 180), (124, 90, 180, 180)])
def test_records_equal_the_per_stage_method(cuda, h, w, nrho, ntheta, dtype):
    check(plan(h, w, nrho, ntheta), patterns(21, h, w, dtype, 900 + h + w))


@pytest.mark.parametrize("h", [200, 240, 252])
def test_large_patterns(cuda, h):
    check(plan(h, h, int(1.5 * h), nbands=10), patterns(5, h, h, np.uint16, 40 + h))


@pytest.mark.parametrize("n", [1, 7, 8, 9, 37, 305, 5000])
def test_pattern_counts(cuda, n):
    check(plan(60, 60, 90, nbands=8), np.resize(patterns(64, 60, 60, np.uint8, 3), (n, 60, 60)))


@pytest.mark.parametrize("frac,mask", [(-0.2, True), (0.0, True), (1.5, True), (0.1, False)])
def test_radon_masks(cuda, frac, mask):
    """Radon masks that change with theta (rays that touch a circle) and ones that do not."""
    check(plan(64, 80, 96, frac=frac, mask=mask), patterns(19, 64, 80, np.uint8, 77))


@pytest.mark.parametrize("dtype", [np.uint8, np.uint16])
def test_degenerate_patterns(cuda, dtype):
    """Ties everywhere (constant images), nothing at all (zeros), saturated images, one bright pixel,
    a checkerboard: more equal candidates than the peak search lists, or fewer peaks than bands."""
    top = np.iinfo(dtype).max
    pats = np.zeros((6, 80, 80), dtype)
    pats[1], pats[2] = 7, top
    pats[3, 40, 41] = top
    pats[4, ::2, ::2] = top
    pats[5, :, :40] = 9
    check(plan(80, 80, 120, nbands=12), pats)
    check(plan(80, 80, 120, nbands=32, mask=False), pats)


def test_one_plan_on_two_streams(cuda):
    """A plan's scratch passes from stream to stream: two streams in turn give one stream's records."""
    import torch
    bd = plan(80, 80, 120)
    dp = bd._device_plan()
    pats = [torch.from_numpy(patterns(700, 80, 80, np.uint8, 10 + k)).to(cuda) for k in range(2)]
    want = [bd.find_bands(p) for p in pats]
    outs = [{f: torch.empty((700, 9, 2) if f in ("maxloc", "aveloc") else (700, 9), device=cuda,
                            dtype=torch.int8 if f == "valid" else torch.float32) for f in _lib.BAND_FIELDS} for _ in pats]
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream(cuda) for _ in pats]
    for _ in range(4):
        for p, o, s in zip(pats, outs, streams):
            dp.find_bands_device(p.data_ptr(), _lib.EBSD_U8, 700, {f: v.data_ptr() for f, v in o.items()}, "fused",
                                 stream=s.cuda_stream)
    torch.cuda.synchronize()
    for o, w in zip(outs, want):
        for f in _lib.BAND_FIELDS:
            assert o[f].cpu().numpy().tobytes() == np.ascontiguousarray(w[f]).tobytes(), f
