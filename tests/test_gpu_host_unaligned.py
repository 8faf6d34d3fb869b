"""Host patterns whose address is no multiple of their type's size (a typed view into a byte buffer):
they are staged, pageable or pinned, in every mode of the host input, and give the records of an
aligned copy.  Reading them in place is not an option: a kernel's load of a pixel has to be aligned."""
import numpy as np
import pytest

import pyebsdindex_gb300 as pg
from pyebsdindex_gb300 import synthetic as syn

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pinned", [False, True])
@pytest.mark.parametrize("dtype,byte", [(np.uint16, 1), (np.uint16, 3), (np.float32, 1), (np.float32, 2)])
@pytest.mark.parametrize("n", [1, 37])
def test_unaligned_input_equals_an_aligned_copy(cuda, n, dtype, byte, pinned):
    import torch
    h = w = 60
    bd = pg.BandDetect(nTheta=180, nRho=90, nBands=8, tSigma=1.0, rSigma=1.0, rhoMaskFrac=0.1)
    bd.band_detect_setup(patDim=(h, w), patternmask=syn.circular_mask(h, w))
    want = syn.make_patterns(n, h, w, seed=5 + n, dtype=np.uint16, peak=4000.0, noise_frac=0.2)[0].astype(dtype)
    buf = torch.empty(want.nbytes + 16, dtype=torch.uint8, pin_memory=pinned).numpy()
    start = (byte - buf.ctypes.data) % 16
    pats = buf[start:start + want.nbytes].view(dtype).reshape(n, h, w)
    pats[...] = want
    assert pats.ctypes.data % 16 == byte and not pats.flags.aligned
    ref = np.array(bd.find_bands(want))
    plan = bd._device_plan()
    for mode in (-1, 0, 1):
        plan.set_host_input(mode)
        got = np.array(bd.find_bands(pats))
        assert got.tobytes() == ref.tobytes(), mode
