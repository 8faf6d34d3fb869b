"""The blocked blur kernel takes batches of many lines, a thread per output the small ones: every output's sum
runs over the same taps in the same order in both, so a batch equals its patterns taken a few at a time bit
for bit.  Line lengths around the group and tile sizes and radii at both ends, batches on either side of
the rule's block counts, and a value that is not finite."""
import numpy as np
import pytest

from pyebsdindex_gb300 import diff

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("h,w,r", [(4, 5, 3), (7, 9, 3), (8, 16, 7), (61, 60, 11), (61, 60, 12), (33, 31, 30), (40, 64, 16),
                                   (17, 200, 5), (13, 12, 4), (300, 6, 4)])
@pytest.mark.parametrize("axis", [0, 1])
@pytest.mark.parametrize("adjoint", [False, True])
def test_batch_equals_parts(cuda, h, w, r, axis, adjoint):
    import torch
    r = min(r, (h if axis == 0 else w) - 1)
    across = w if axis == 0 else h                # lines of a pattern
    least = 32 * (152 if r < 12 else 64)          # the rule's blocks of 32 lines
    lib, g = diff._bind(), np.random.default_rng(h * w)
    taps = torch.from_numpy(g.normal(size=2 * r + 1).astype(np.float32)).to(cuda)
    for n in (least // across + 3, (least - 32) // across - 1):
        x = torch.from_numpy(g.normal(size=(n, h * w)).astype(np.float32)).to(cuda)
        x[n // 2, (h // 2) * w + w // 2] = float("inf")
        step = max(1, 512 // across)
        whole = diff._blur(lib, x, taps, r, h, w, axis, adjoint)
        parts = torch.cat([diff._blur(lib, x[s:s + step].contiguous(), taps, r, h, w, axis, adjoint)
                           for s in range(0, n, step)])
        a, b = whole.cpu().numpy(), parts.cpu().numpy()
        assert np.array_equal(np.isfinite(a), np.isfinite(b))
        keep = np.isfinite(a)
        assert np.array_equal(a[keep], b[keep])
        assert (~keep).sum() <= 2 * (2 * r + 1)
