"""Small pageable host input, which the strip kernels read where it lies (one chunk, integer
patterns): the same records as the staged copy of it, for a single pattern, an ordinary chunk,
a read-only array and one that starts at an odd address."""
import numpy as np
import pytest

import pyebsdindex_gb300 as pg
from pyebsdindex_gb300 import synthetic as syn

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", ["uint8", "uint16"])
@pytest.mark.parametrize("n,shift,frozen", [(1, 0, False), (7, 1, False), (528, 0, True), (700, 3, False)])
def test_pageable_input_equals_staged(cuda, n, shift, frozen, dtype):
    h = w = 60
    bd = pg.BandDetect(nTheta=180, nRho=90, nBands=8, tSigma=1.0, rSigma=1.0, rhoMaskFrac=0.1)
    bd.band_detect_setup(patDim=(h, w), patternmask=syn.circular_mask(h, w))
    rng = np.random.default_rng(n)
    buf = np.zeros(n * h * w + shift, dtype)
    buf[shift:] = rng.integers(0, 250, size=n * h * w)
    pats = buf[shift:].reshape(n, h, w)
    if frozen:
        pats.flags.writeable = False
    plan = bd._device_plan()
    out = {}
    for mode in (-1, 0):
        plan.set_host_input(mode)
        out[mode] = np.array(bd.find_bands(pats))
    plan.set_host_input(-1)
    assert out[-1].shape[0] == n and out[-1].tobytes() == out[0].tobytes()
