"""Pinned integer patterns on either side of the size up to which the strip kernels read them in place (1 MB a
call): the same records in every mode of the host input, and as from ordinary memory."""
import numpy as np
import pytest

import pyebsdindex_gb300 as pg
from pyebsdindex_gb300 import synthetic as syn

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [np.uint8, np.uint16])
@pytest.mark.parametrize("size", [3600, (1 << 20) - 3600, (1 << 20) + 7200, 5 << 20])
def test_pinned_input(cuda, size, dtype):
    import torch
    h = w = 60
    n = max(1, size // (h * w * np.dtype(dtype).itemsize))
    bd = pg.BandDetect(nTheta=180, nRho=90, nBands=8, tSigma=1.0, rSigma=1.0, rhoMaskFrac=0.1)
    bd.band_detect_setup(patDim=(h, w), patternmask=syn.circular_mask(h, w))
    src = np.resize(syn.make_patterns(97, h, w, seed=n, dtype=dtype, noise_frac=0.2)[0], (n, h, w))
    pats = torch.empty(src.nbytes, dtype=torch.uint8, pin_memory=True).numpy().view(dtype).reshape(n, h, w)
    pats[...] = src
    want = np.array(bd.find_bands(src))
    plan = bd._device_plan()
    for mode in (-1, 0, 1):
        plan.set_host_input(mode)
        assert np.array(bd.find_bands(pats)).tobytes() == want.tobytes(), mode
