"""The peak kernel of the strip path for every LoG size it takes (rho taps x theta taps: 7x5, which
a default BandDetect has, 5x7, 7x7, 9x9; the other strip tests run 5x5): ring length, padding, float4
count and zero-extended statistics rows differ for each.  Records equal the per-stage method's bit for
bit, normmax (its mean reduced in another order) to 1e-6.  Sizes: one rho segment and several, one theta
slab and several, one pattern and a unit cut short; 9x9 for uint8 where the one-tile kernel does not
take the plan."""
import numpy as np
import pytest

import pyebsdindex_gb300 as pg
from pyebsdindex_gb300 import synthetic as syn

pytestmark = pytest.mark.gpu

FIELDS = ("max", "maxloc", "avemax", "aveloc", "width", "theta", "rho", "valid")
LOG = {(7, 5): (None, None), (5, 7): (1.0, 1.5), (7, 7): (1.5, 1.5), (9, 9): (2.0, 2.0)}


@pytest.mark.parametrize("dtype", [np.uint8, np.uint16])
@pytest.mark.parametrize("taps", list(LOG))
@pytest.mark.parametrize("h,w,nrho,ntheta", [(40, 45, 62, 180), (80, 80, 120, 180), (84, 100, 150, 97), (120, 120, 180, 180),
                                             (240, 240, 360, 180)])
def test_records_equal_the_per_stage_method(cuda, h, w, nrho, ntheta, taps, dtype):
    rs, ts = LOG[taps]
    bd = pg.BandDetect(nTheta=ntheta, nRho=nrho, tSigma=ts, rSigma=rs, rhoMaskFrac=0.1, nBands=9)
    bd.band_detect_setup(patDim=(h, w), patternmask=syn.circular_mask(h, w))
    assert np.shape(bd.kernel)[-2:] == taps
    pats = syn.make_patterns(19 if h < 200 else 5, h, w, seed=h + w, dtype=dtype, peak=200.0 if dtype == np.uint8 else 4000.0,
                             noise_frac=0.2)[0]
    pats[1], pats[2] = 0, 7
    want = bd.find_bands(pats, method="plain")
    for sel in (slice(None), slice(0, 1)):
        got = bd.find_bands(pats[sel], method="fused")
        for f in FIELDS:
            assert got[f].tobytes() == want[sel][f].tobytes(), f
        np.testing.assert_allclose(got["normmax"], want[sel]["normmax"], rtol=1e-6)
