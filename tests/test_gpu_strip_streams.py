"""One plan's scratch between streams of one handle: per-thread default streams of two host threads, and a
stream destroyed while its work runs whose handle the next stream may take again.  Each call waits for the
one before it on the device, so every call gives the records of a call alone."""
import ctypes as C
import threading

import numpy as np
import pytest

import pyebsdindex_gb300 as pg
from pyebsdindex_gb300 import _lib, synthetic as syn

pytestmark = pytest.mark.gpu
N = 1500


def setup(cuda, count):
    import torch
    bd = pg.BandDetect(nTheta=180, nRho=120, tSigma=1.0, rSigma=1.0, rhoMaskFrac=0.1, nBands=9)
    bd.band_detect_setup(patDim=(80, 80), patternmask=syn.circular_mask(80, 80))
    pats = [torch.from_numpy(syn.make_patterns(N, 80, 80, seed=60 + k, noise_frac=0.2)[0]).to(cuda) for k in range(count)]
    want = [bd.find_bands(p) for p in pats]
    outs = [{f: torch.empty((N, 9, 2) if f in ("maxloc", "aveloc") else (N, 9), device=cuda,
                            dtype=torch.int8 if f == "valid" else torch.float32) for f in _lib.BAND_FIELDS} for _ in pats]
    torch.cuda.synchronize()
    return bd._device_plan(), pats, outs, want


def call(dp, pats, out, stream):
    dp.find_bands_device(pats.data_ptr(), _lib.EBSD_U8, N, {f: v.data_ptr() for f, v in out.items()}, "fused", stream=stream)


def check(outs, want):
    import torch
    torch.cuda.synchronize()
    for o, w in zip(outs, want):
        for f in _lib.BAND_FIELDS:
            assert o[f].cpu().numpy().tobytes() == np.ascontiguousarray(w[f]).tobytes(), f


def test_per_thread_streams(cuda):
    dp, pats, outs, want = setup(cuda, 2)
    per_thread = 2  # cudaStreamPerThread
    errors = []

    def work(k):
        try:
            for _ in range(8):
                call(dp, pats[k], outs[k], per_thread)
        except Exception as e:  # noqa: BLE001
            errors.append(e)
    threads = [threading.Thread(target=work, args=(k,)) for k in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors
    check(outs, want)


def test_a_handle_used_again(cuda):
    import torch
    rt = torch.cuda.cudart()
    dp, pats, outs, want = setup(cuda, 4)
    for p, o in zip(pats, outs):
        h = C.c_void_p()
        assert int(rt.cudaStreamCreate(C.addressof(h))) == 0
        call(dp, p, o, h.value)
        assert int(rt.cudaStreamDestroy(h.value)) == 0
    check(outs, want)
