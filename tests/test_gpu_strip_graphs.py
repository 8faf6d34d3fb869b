"""Captured calls of the strip path have scratch of their graph's own: graphs of one plan replayed at once,
beside direct calls of the plan, give the records of calls alone; the buffer of a graph that is gone
serves the next capture; a plan's first call may be a captured one; and a plan that allocates while some
other stream is captured leaves that capture alone."""
import time

import numpy as np
import pytest

import pyebsdindex_gb300 as pg
from pyebsdindex_gb300 import _lib, synthetic as syn

pytestmark = pytest.mark.gpu
CODE = {"uint8": _lib.EBSD_U8, "uint16": _lib.EBSD_U16}


def plan():
    bd = pg.BandDetect(nTheta=180, nRho=120, tSigma=1.0, rSigma=1.0, rhoMaskFrac=0.1, nBands=9)
    bd.band_detect_setup(patDim=(80, 80), patternmask=syn.circular_mask(80, 80))
    return bd


class Call:
    """n patterns on the device, their outputs, and the records that a call alone gives."""

    def __init__(self, cuda, n, seed, dtype="uint8"):
        import torch
        host = syn.make_patterns(n, 80, 80, seed=seed, dtype=np.dtype(dtype), noise_frac=0.2)[0]
        self.n, self.dt = n, CODE[dtype]
        self.pats = torch.from_numpy(host.view(np.uint8).reshape(n, -1)).to(cuda)
        self.outs = {f: torch.zeros((n, 9, 2) if f in ("maxloc", "aveloc") else (n, 9), device=cuda,
                                    dtype=torch.int8 if f == "valid" else torch.float32) for f in _lib.BAND_FIELDS}
        self.want = plan().find_bands(host, method="fused")

    def run(self, dp, stream):
        dp.find_bands_device(self.pats.data_ptr(), self.dt, self.n, {f: v.data_ptr() for f, v in self.outs.items()},
                             "fused", stream=stream.cuda_stream)

    def check(self):
        for f in _lib.BAND_FIELDS:
            assert self.outs[f].cpu().numpy().tobytes() == np.ascontiguousarray(self.want[f]).tobytes(), f


def capture(dp, calls):
    import torch
    g, s = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.graph(g, stream=s):
        for c in calls:
            c.run(dp, s)
    return g


@pytest.mark.parametrize("dtype", ["uint8", "uint16"])
@pytest.mark.parametrize("n", [3, 700, 3000])
def test_graphs_of_one_plan_at_once(cuda, n, dtype):
    import torch
    dp = plan()._device_plan()
    calls = [Call(cuda, n, 10 + k, dtype) for k in range(5)]
    graphs = [capture(dp, calls[0:1]), capture(dp, calls[1:3]), capture(dp, calls[3:4])]  # the first on a fresh plan
    streams = [torch.cuda.Stream() for _ in range(4)]
    for rep in range(5):
        for c in calls:
            for v in c.outs.values():
                v.zero_()
        torch.cuda.synchronize()
        for g, s in zip(graphs, streams):
            with torch.cuda.stream(s):
                g.replay()
        calls[4].run(dp, streams[3])
        torch.cuda.synchronize()
        for c in calls:
            c.check()


def test_the_buffer_of_a_graph_that_is_gone_serves_the_next(cuda):
    import torch
    dp = plan()._device_plan()
    call = Call(cuda, 2000, 3)

    def used():
        torch.cuda.synchronize()
        free, total = torch.cuda.mem_get_info()
        return total - free
    sizes = []
    for _ in range(6):
        g = capture(dp, [call])
        g.replay()
        torch.cuda.synchronize()
        call.check()
        g.reset()
        del g
        time.sleep(0.5)  # the runtime drops what the graph held on a thread of its own
        sizes.append(used())
    assert sizes[-1] - sizes[1] < 16 << 20, sizes  # a buffer of 2,000 patterns takes more than 200 MB


def test_allocating_beside_a_capture(cuda):
    import torch
    call, other = Call(cuda, 300, 5), Call(cuda, 500, 6)
    dp, fresh = plan()._device_plan(), plan()._device_plan()
    g, s, t = torch.cuda.CUDAGraph(), torch.cuda.Stream(), torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.graph(g, stream=s):
        call.run(dp, s)
        other.run(fresh, t)  # not captured: the plan's first call allocates its scratch
    g.replay()
    torch.cuda.synchronize()
    call.check()
    other.check()
