"""A pinned tile shape takes integer calls off the strip kernels: the one-tile kernel in every pass width,
theta slabs of several counts and the mixed-size launch give the per-stage method's records for uint8
and uint16 patterns bit for bit (normmax, whose mean each kernel reduces in its own order, to 1e-6), and the
launch counts say which kernels ran (strip: four a pass; one tile or slabs: two; a mixed launch: one, and one
a size)."""
import json

import numpy as np
import pytest

import pyebsdindex_gb300 as pg
from pyebsdindex_gb300 import _lib, synthetic as syn
from pyebsdindex_gb300.band_detect import MixedBandDetect

pytestmark = pytest.mark.gpu

FIELDS = ("max", "maxloc", "avemax", "aveloc", "width", "theta", "rho", "valid")
CODE = {"uint8": _lib.EBSD_U8, "uint16": _lib.EBSD_U16}


def plan(h, nrho, nbands=9):
    bd = pg.BandDetect(nTheta=180, nRho=nrho, tSigma=1.0, rSigma=1.0, rhoMaskFrac=0.1, nBands=nbands)
    bd.band_detect_setup(patDim=(h, h), patternmask=syn.circular_mask(h, h))
    return bd


def patterns(n, h, dtype, seed):
    p = syn.make_patterns(n, h, h, seed=seed, dtype=np.dtype(dtype), peak=200.0 if dtype == "uint8" else 4000.0, noise_frac=0.2)[0]
    p[1], p[2] = 0, 7  # nothing, and ties everywhere
    return p


def same(a, b):
    for f in FIELDS:
        assert a[f].tobytes() == b[f].tobytes(), f
    np.testing.assert_allclose(a["normmax"], b["normmax"], rtol=1e-6)


@pytest.mark.parametrize("dtype", ["uint8", "uint16"])
@pytest.mark.parametrize("h,nrho", [(60, 90), (80, 120), (120, 180)])
def test_pinned_shapes(cuda, h, nrho, dtype):
    bd = plan(h, nrho)
    dp = bd._device_plan()
    info = dp.get_tile()
    pats = patterns(203, h, dtype, h)
    ref = bd.find_bands(pats, method="plain")
    strip = bd.find_bands(pats, method="fused")
    assert dp.strip_serves("fused", CODE[dtype]) and dp.last_launches() == 4
    shapes = [(2, ns) for ns in range(info["slabs_min"], min(info["slabs_max"], info["slabs_min"] + 2) + 1)]
    if info["single_fits"]:
        shapes.append((1, 0))
    assert shapes
    for shape in shapes:
        dp.set_tile(*shape)
        assert not dp.strip_serves("fused", CODE[dtype])
        widths = []
        for ppp in (1, 2, 4, 8, 0) if shape[0] == 1 else (0,):
            dp.set_patterns_per_pass(ppp)
            rec = bd.find_bands(pats, method="fused")
            assert dp.last_launches() == 2
            same(rec, ref)
            widths.append(rec.tobytes())
        assert len(set(widths)) == 1
        parts = np.concatenate([bd.find_bands(pats[s:s + 7], method="fused") for s in range(0, 203, 7)])
        assert parts.tobytes() == widths[0]
    dp.set_tile(0, 0)
    assert dp.strip_serves("fused", CODE[dtype])
    assert bd.find_bands(pats, method="fused").tobytes() == strip.tobytes() and dp.last_launches() == 4


@pytest.mark.parametrize("dtype", ["uint8", "uint16"])
def test_mixed_sizes_in_one_launch(cuda, dtype):
    import torch
    mb = MixedBandDetect(nBands=10, mask_for=syn.circular_mask)
    host = {(h, h): patterns(n, h, dtype, 40 + h) for h, n in ((60, 301), (120, 77), (240, 19))}
    dev = {k: torch.from_numpy(v.view(np.int16 if dtype == "uint16" else np.uint8)).to(cuda) for k, v in host.items()}
    if dtype == "uint16":
        if not hasattr(torch, "uint16"):
            pytest.skip("torch without uint16")
        dev = {k: v.view(torch.uint16) for k, v in dev.items()}
    plans = {k: mb.plan(*k)._device_plan() for k in host}

    def run(out=None, stream=None):
        out = mb.find_bands_device(dev, out=out, stream=stream)
        assert mb.last_mixed
        return out

    def numpy(out):
        torch.cuda.synchronize()
        return {k: {f: v.cpu().numpy() for f, v in o.items()} for k, o in out.items()}

    strip = numpy(run())
    assert plans[(60, 60)].last_launches() == 12
    plans[(120, 120)].set_tile(2, 0)  # one pinned plan takes the whole call
    out = run()
    assert plans[(60, 60)].last_launches() == 4
    slabs = numpy(out)
    for k in host:
        same(slabs[k], strip[k])
        same(slabs[k], mb.plan(*k).find_bands(host[k], method="plain"))
    # and captured
    side, g = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    side.wait_stream(torch.cuda.current_stream())
    for o in out.values():
        for v in o.values():
            v.zero_()
    torch.cuda.synchronize()
    with torch.cuda.graph(g, stream=side):
        run(out, side)
    g.replay()
    again = numpy(out)
    for k in host:
        for f in _lib.BAND_FIELDS:
            assert again[k][f].tobytes() == slabs[k][f].tobytes(), (k, f)


def test_autotune_ends_a_pin(cuda):
    import torch
    bd = plan(60, 90)
    dp = bd._device_plan()
    pats = patterns(64, 60, "uint8", 4)
    dp.set_tile(1, 0)
    assert not dp.strip_serves("fused", _lib.EBSD_U8)
    assert bd.autotune(torch.from_numpy(pats), method="fused") == 8
    assert dp.strip_serves("fused", _lib.EBSD_U8)
    # what is chosen for float patterns leaves integer ones where they are
    bd.autotune(torch.from_numpy(pats.astype(np.float32)), method="fused")
    assert dp.strip_serves("fused", _lib.EBSD_U8) and not dp.strip_serves("fused", _lib.EBSD_F32)
    bd.find_bands(pats, method="fused")
    assert dp.last_launches() == 4


@pytest.mark.parametrize("tile", [None, 1, 2])
def test_a_stored_decision_pins_nothing_for_integers(cuda, tmp_path, tile):
    """Decisions stored by a library that timed integer patterns' tiles."""
    import torch
    from pyebsdindex_gb300 import tuning
    path = tmp_path / "tuning.json"
    pats = patterns(64, 60, "uint8", 4)
    first = plan(60, 90)
    first.autotune(torch.from_numpy(pats), method="fused", cache=path)
    key = next(iter(json.loads(path.read_text())["entries"]))
    entry = {"patterns_per_pass": 1 if tile == 2 else 4}
    if tile:
        entry.update(tile=tile, slabs=first._device_plan().get_tile()["slabs_min"] + 1 if tile == 2 else 0)
    tuning.TuningCache(path).put(key, entry)
    bd = plan(60, 90)
    assert bd.autotune(torch.from_numpy(pats), method="fused", cache=path) == entry["patterns_per_pass"] and bd.tuned["cached"]
    dp = bd._device_plan()
    if tile == 2:
        assert dp.get_tile()["slabs"] == entry["slabs"]
    rec = bd.find_bands(pats, method="fused")
    assert dp.strip_serves("fused", _lib.EBSD_U8) and dp.last_launches() == 4
    assert rec.tobytes() == first.find_bands(pats, method="fused").tobytes()
