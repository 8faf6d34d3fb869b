"""The pair kernel with saturated values: pixels that hold one are summed term by term, the others whole, so
the sums are those of the kernels that test every term, bit for bit, from a few saturated values to patterns of
nothing else, with a NaN, and with pixel lists that leave a short last chunk."""
import numpy as np
import pytest

from pyebsdindex_gb300 import diff

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nr,nc,npx,nind,sr", [(5, 64, 200, 200, 1), (9, 130, 130, 97, 2), (12, 61, 96, 70, 3), (7, 7, 333, 301, 3),
                                               (6, 122, 64, 33, 1)])
@pytest.mark.parametrize("share", [0.0002, 0.01, 0.3, 1.0])
def test_sums_equal_the_kernels_that_test_every_term(cuda, nr, nc, npx, nind, sr, share):
    import torch
    from pyebsdindex_gb300 import _lib
    lib, g, n, ws = diff._bind(), np.random.default_rng(int(1e4 * share) + npx), nr * nc, (2 * sr + 1) ** 2
    x = (g.random((n, npx)) * 190.0).astype(np.float32)
    x[g.random(x.shape) < share] = 199.5          # between the levels of the weights (0.999) and of sigma (0.9961)
    x[g.random(x.shape) < share / 2] = 200.0      # beyond both
    x[n // 3, npx // 2] = np.nan
    xt = torch.from_numpy(x).to(cuda)
    ind = torch.from_numpy(np.sort(g.permutation(npx)[:nind]).astype(np.int32)).to(cuda)
    st = torch.cuda.current_stream().cuda_stream

    def outs():
        return [torch.zeros(n, device=cuda), torch.zeros(n, dtype=torch.int32, device=cuda), torch.zeros(n, device=cuda)] + [
            torch.zeros((n, ws), device=cuda) for _ in range(4)]
    a, b = outs(), outs()
    head = (xt.data_ptr(), nr, nc, npx, ind.data_ptr(), nind, 200.0)
    _lib.check(lib.ebsd_nlpar_sigma_arg(*head, 1, *(t.data_ptr() for t in a[:3]), st), "sigma_arg")
    _lib.check(lib.ebsd_nlpar_weights_d(*head, 0.9, sr, 0.1, a[0].data_ptr(), 1, *(t.data_ptr() for t in a[3:]), st), "weights_d")
    work = torch.empty(int(lib.ebsd_nlpar_sigma_weights_d_work(nr, nc, sr)), device=cuda)
    _lib.check(lib.ebsd_nlpar_sigma_weights_d(*head, 0.9, sr, 0.1, 1, 1, work.data_ptr(), *(t.data_ptr() for t in b), st),
               "sigma_weights_d")
    for s, t in zip(a, b):
        assert torch.equal(s.view(torch.int32), t.view(torch.int32))
