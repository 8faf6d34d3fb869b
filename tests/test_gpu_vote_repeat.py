"""Votes over a library whose rows repeat: every match is counted once a copy, so the vote counts are the
copies times those of one copy, exactly and for every pattern (a vote on the edge of its tolerance falls on
the same side in each copy).  Lists that fill, that are cut, and single band triplets with more matches
than a list holds."""
import os

import numpy as np
import pytest

from conftest import GOLDEN_DIR
from oracle import vote_oracle as vo

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("copies,nb", [(2, 9), (12, 8), (13, 3), (41, 6), (90, 5), (159, 4), (160, 4), (161, 4), (300, 4)])
def test_counts_are_the_copies_times_one(cuda, copies, nb):
    import torch
    from pyebsdindex_gb300 import tripletvote as tv
    lib, params, ins, _ = vo.load_case(os.path.join(GOLDEN_DIR, "vote_fcc_syn.npz"))
    norms, inten = ins["norms"][:200, :nb].copy(), ins["inten"][:200, :nb].copy()
    inten[5, nb // 2] = 0.0
    keep = max(1, min(len(lib["trip_angles"]), 7000 // copies))

    def counts(times):
        l = dict(lib)
        for k in ("trip_angles", "trip_familyid"):
            l[k] = np.tile(lib[k][:keep], (times, 1))
        bi = tv.BandIndexer(lib=l, angTol=params["angTol"], nband_earlyexit=params["nband_earlyexit"],
                            simpleqweights=params["simpleqweights"], high_fidelity=True)
        out = bi.bandindex_device(torch.from_numpy(norms).cuda(), torch.from_numpy(inten).cuda(), intermediates=True)
        return out["accn"].cpu().numpy(), out["accw"].cpu().numpy()

    (n1, w1), (nc, wc) = counts(1), counts(copies)
    assert n1.sum() > 0
    assert np.array_equal(nc, n1 * copies)
    # the weights: a float32 sum of all counts' terms, each between 0 and the tolerance
    terms = nc.astype(np.float64)
    assert np.all(np.abs(wc - copies * w1.astype(np.float64)) <= (terms + 2) * 2.0 ** -24 * terms * params["angTol"] + 1e-30)
