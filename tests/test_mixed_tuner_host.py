"""The mixed-size tuner, without a GPU: where the strip kernels serve every size of the batch no slab count is
timed and the plans stay as they are; with one size that they do not serve, every size is timed in slabs."""
import pytest

from pyebsdindex_gb300.band_detect import MixedBandDetect


class FakePlan:
    device = 0

    def __init__(self, strips):
        self.strips, self.calls, self.pinned = strips, [], 0

    def strip_serves(self, method, dtype):
        return self.strips and not self.pinned

    def set_tile(self, tile, slabs=0):
        self.calls.append((tile, slabs))
        self.pinned = tile

    def get_tile(self):
        return {"tile": 1, "slabs": 9, "slabs_min": 9, "slabs_max": 11}

    def supported(self, method, dtype=None):
        return True

    def find_bands_device(self, *a, **k):
        raise AssertionError("timed")


@pytest.mark.parametrize("served", [True, False])
def test_mixed_tuner(monkeypatch, served):
    torch = pytest.importorskip("torch")
    mb = MixedBandDetect(nBands=10)
    plans = {(60, 60): FakePlan(True), (120, 120): FakePlan(served)}
    monkeypatch.setattr(mb, "plan", lambda h, w: type("B", (), {"_device_plan": lambda self: plans[(h, w)]})())
    monkeypatch.setattr(torch.cuda, "current_stream", lambda dev=None: type("S", (), {"cuda_stream": 0})())
    monkeypatch.setattr(torch.cuda, "Event", lambda **k: type("E", (), {"record": lambda self, st: None})())
    import pyebsdindex_gb300.band_detect as band_detect
    monkeypatch.setattr(band_detect, "_device_input", lambda t, dev: (t, 0))
    monkeypatch.setattr(mb, "_device_outputs", lambda n, dev: {})
    batches = {k: torch.zeros((3,) + k, dtype=torch.uint8) for k in plans}
    if served:
        assert mb.autotune(batches) == {k: {"slabs": 9, "ms": {}} for k in plans}
        assert all(p.calls == [] for p in plans.values())
    else:
        with pytest.raises(AssertionError, match="timed"):  # every size is timed in slabs
            mb.autotune(batches)
