"""Host logic around the strip kernels, without a GPU: a stored tuning decision for integer patterns re-lays the
slab tables and pins no tile shape where the strip kernels serve the call, and pins it where they do not."""
import pytest

import pyebsdindex_gb300 as pg


class FakePlan:
    device = 0

    def __init__(self, strips, slabs_max=11):
        self.strips, self.calls, self.ppp, self.slabs_max, self.slabs, self.pinned = strips, [], None, slabs_max, 9, 0

    def strip_serves(self, method, dtype):
        return self.strips and not self.pinned and dtype in (0, 1)

    def set_tile(self, tile, slabs=0):
        if slabs > self.slabs_max:
            raise RuntimeError("ebsd_plan_set_tile failed: plan shape not supported by this method (code -5)")
        self.calls.append((tile, slabs))
        self.pinned, self.slabs = tile, slabs or 9

    def set_patterns_per_pass(self, ppp):
        self.ppp = ppp

    def get_tile(self):
        return {"tile": 1, "slabs": self.slabs, "slabs_min": 9, "slabs_max": self.slabs_max, "patterns_per_pass": self.ppp}

    def supported(self, method, dtype=None):
        return True

    def autotune(self, *a, **k):
        raise AssertionError("timed")


@pytest.mark.parametrize("strips", [True, False])
@pytest.mark.parametrize("entry", [{"patterns_per_pass": 8, "tile": 1, "slabs": 0}, {"patterns_per_pass": 1, "tile": 2, "slabs": 10},
                                   {"patterns_per_pass": 4}])
@pytest.mark.parametrize("dtype", ["uint8", "float32"])
def test_stored_decision(tmp_path, monkeypatch, strips, entry, dtype):
    torch = pytest.importorskip("torch")
    from pyebsdindex_gb300 import tuning
    bd = pg.BandDetect(patDim=(60, 60), nRho=90, nTheta=180, tSigma=1.0, rSigma=1.0, nBands=10)
    plan = FakePlan(strips)
    monkeypatch.setattr(bd, "_device_plan", lambda gpu_id=None: plan)
    monkeypatch.setattr(bd, "_tuning_key", lambda p, m, dt: "key")
    path = tmp_path / "tuning.json"
    tuning.TuningCache(path).put("key", entry)
    sample = torch.zeros((4, 60, 60), dtype=getattr(torch, dtype))
    assert bd.autotune(sample, method="fused", cache=path) == entry["patterns_per_pass"]
    assert bd.tuned["cached"] and plan.ppp == entry["patterns_per_pass"]
    on_strips = strips and dtype == "uint8"
    assert plan.pinned == (0 if on_strips else entry.get("tile", 0))
    assert plan.slabs == (10 if entry.get("tile") == 2 else 9)
