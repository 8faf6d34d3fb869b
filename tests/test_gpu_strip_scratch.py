"""The strip path's scratch is as large as the calls need: a plan that has detected one pattern holds a
small part of what a whole pass takes, a larger call grows it, and the records do not depend on it."""
import numpy as np
import pytest

import pyebsdindex_gb300 as pg
from pyebsdindex_gb300 import synthetic as syn

pytestmark = pytest.mark.gpu


def plan():
    bd = pg.BandDetect(nTheta=180, nRho=120, tSigma=1.0, rSigma=1.0, rhoMaskFrac=0.1, nBands=9)
    bd.band_detect_setup(patDim=(80, 80), patternmask=syn.circular_mask(80, 80))
    return bd


def used(torch):
    torch.cuda.synchronize()
    free, total = torch.cuda.mem_get_info()
    return total - free


def test_scratch_grows_with_the_calls(cuda):
    import torch
    pats = syn.make_patterns(5000, 80, 80, seed=8, noise_frac=0.2)[0]
    first = plan()  # (kept: loads the kernels, and frees nothing below)
    want = first.find_bands(pats, method="fused")
    bd = plan()
    bd._device_plan()
    before = used(torch)
    recs = [bd.find_bands(pats[:1], method="fused")]
    one = used(torch) - before
    for n in (100, 65, 700, 5000, 129):
        recs.append(bd.find_bands(pats[:n], method="fused"))
    many = used(torch) - before
    print("one pattern: %.1f MB, 5000: %.1f MB" % (one / 2 ** 20, many / 2 ** 20))
    assert one < 64 << 20  # 64 patterns of 0.12 MB and the call's own buffers, against 0.3 GB for a whole pass
    for r in recs:
        assert r.tobytes() == want[:len(r)].tobytes()


def test_reserve_then_no_allocation(cuda):
    import torch
    from pyebsdindex_gb300 import _lib
    n = 3000
    pats = torch.from_numpy(syn.make_patterns(n, 80, 80, seed=9, noise_frac=0.2)[0]).to(cuda)
    outs = {f: torch.empty((n, 9, 2) if f in ("maxloc", "aveloc") else (n, 9), device=cuda,
                           dtype=torch.int8 if f == "valid" else torch.float32) for f in _lib.BAND_FIELDS}
    first = plan()
    first.find_bands(pats[:200], method="fused")
    bd = plan()
    dp = bd._device_plan()
    dp.reserve("fused", n)
    before = used(torch)
    for m in (1, 800, n):
        dp.find_bands_device(pats.data_ptr(), _lib.EBSD_U8, m, {f: v.data_ptr() for f, v in outs.items()}, "fused",
                             stream=torch.cuda.current_stream().cuda_stream)
    assert used(torch) == before


def test_growing_beside_a_capture(cuda):
    import torch
    from pyebsdindex_gb300 import _lib
    host = syn.make_patterns(2000, 80, 80, seed=11, noise_frac=0.2)[0]
    pats = torch.from_numpy(host).to(cuda)
    a, b = plan(), plan()
    want = a.find_bands(host, method="fused")

    def call(bd, n, stream, out):
        bd._device_plan().find_bands_device(pats.data_ptr(), _lib.EBSD_U8, n, {f: v.data_ptr() for f, v in out.items()},
                                            "fused", stream=stream.cuda_stream)

    def outs():
        return {f: torch.zeros((2000, 9, 2) if f in ("maxloc", "aveloc") else (2000, 9), device=cuda,
                               dtype=torch.int8 if f == "valid" else torch.float32) for f in _lib.BAND_FIELDS}
    oa, ob = outs(), outs()
    g, s, t = torch.cuda.CUDAGraph(), torch.cuda.Stream(), torch.cuda.Stream()
    torch.cuda.synchronize()
    call(b, 10, t, ob)
    t.synchronize()
    with torch.cuda.graph(g, stream=s):
        call(a, 2000, s, oa)
        call(b, 2000, t, ob)  # not captured: a larger scratch takes the place of the first
    g.replay()
    torch.cuda.synchronize()
    for o in (oa, ob):
        for f in _lib.BAND_FIELDS:
            assert o[f].cpu().numpy().tobytes() == np.ascontiguousarray(want[f]).tobytes(), f
