"""The soft-argmax of float patterns forms the exponents and the gradient in double: where one cell is
all of the softmax (every other exponent below -200, whose float exponential is zero) its gradient
s (1 + (c - J) / tau) is 1 and J is the cell's value, whatever c / tau is.  J = (1 v) / 1 is exact
in double, so c - J is zero; the largest exponent is c / tau less its own rounded product, at most
2^-53 |c / tau| < 2^-24, whose exponential rounds to 1."""
import numpy as np
import pytest

from pyebsdindex_gb300 import diff

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tau", [1e-6, 3e-6, 1.1e-5, 7e-4])
@pytest.mark.parametrize("sign", [1.0, -1.0])
def test_one_dominant_cell_has_gradient_one(cuda, tau, sign):
    import torch
    from pyebsdindex_gb300 import _lib
    n, ncell = 64, 700
    g = np.random.default_rng(int(1e7 * tau))
    top = sign * (100.0 + 100.0 * g.random(n))
    c = (top[:, None] - 1.0 - 10.0 * g.random((n, ncell))).astype(np.float32)
    at = g.integers(0, ncell, size=n)
    c[np.arange(n), at] = top
    ct = torch.from_numpy(c).to(cuda)
    ci = torch.arange(ncell, dtype=torch.int32, device=cuda)
    J, grad = torch.empty(n, dtype=torch.float64, device=cuda), torch.zeros_like(ct)
    _lib.check(diff._bind().ebsd_softargmax(0, ct.data_ptr(), n, ncell, ci.data_ptr(), ncell, tau, J.data_ptr(),
                                            grad.data_ptr(), torch.cuda.current_stream().cuda_stream), "softargmax")
    want = np.zeros((n, ncell), np.float32)
    want[np.arange(n), at] = 1.0
    assert np.array_equal(J.cpu().numpy(), c[np.arange(n), at].astype(np.float64))
    assert np.array_equal(grad.cpu().numpy(), want)
