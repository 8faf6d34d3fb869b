"""normmax of dim integer patterns on the strip path: a flat background of a few counts with one pixel
a count above it.

The flat part convolves to the rounding residue of the taps' sum, the same small value in nearly every
cell, so a rounding that is coarse beside it does not average out of the mean that normmax divides by.
The per-stage method sums the mean in double.  The strip path adds four cells in float, which is exact
for four equal ones (x + x, 3x + x: the rounding of 3x is at most a quarter of 4x's spacing), so only the
cells under the pixel's curve round: some 500 sums of at most 0.1, at random 2^-25 x 0.1 x 22 = 7e-8 in a sum
over 18,000 cells or more, 1e-10 of mean - min (0.03), against a spacing of 6e-8 at least: other bits than the
per-stage method's in well below one pattern of a hundred."""
import numpy as np
import pytest

import pyebsdindex_gb300 as pg
from pyebsdindex_gb300 import synthetic as syn

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [np.uint8, np.uint16])
@pytest.mark.parametrize("h,nrho,sigma", [(80, 120, None), (60, 90, 1.2), (80, 120, 1.0), (120, 180, 1.2)])
def test_normmax_of_dim_patterns(cuda, h, nrho, sigma, dtype):
    bd = pg.BandDetect(nTheta=180, nRho=nrho, tSigma=sigma, rSigma=sigma, rhoMaskFrac=0.1, nBands=2)
    bd.band_detect_setup(patDim=(h, h), patternmask=syn.circular_mask(h, h))
    g = np.random.default_rng(h)
    n = 600
    pats = np.zeros((n, h, h), dtype)
    pats += (1 + np.arange(n) % 3)[:, None, None].astype(dtype)
    at = h // 2 + g.integers(-h // 4, h // 4, size=(2, n))
    pats[np.arange(n), at[0], at[1]] += dtype(1)
    want, got = bd.find_bands(pats, method="plain"), bd.find_bands(pats, method="fused")
    assert want["max"].tobytes() == got["max"].tobytes()
    a, b = want["normmax"][:, 0].copy(), got["normmax"][:, 0].copy()
    differ = np.abs(a.view(np.int32) - b.view(np.int32))
    print(h, sigma, np.dtype(dtype).name, "differing %.3f, by %d at most" % ((differ > 0).mean(), differ.max()))
    assert (differ > 0).mean() <= 0.01
