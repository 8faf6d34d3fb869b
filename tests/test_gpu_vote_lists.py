"""The vote's match lists and the grouped TRIAD candidates at their edges, against the oracle: band
counts that leave lanes over or fill the warp, libraries whose rows repeat so that 32 band triplets'
matches need several lists, or one band triplet more than a list holds.

A pattern may differ where a vote or a tolerance test sits on its edge (the arccos of the two sides
differ in the last bits): nine in ten must agree in every integer, and there the weighted votes to
1e-5, as in the golden tests."""
import os

import numpy as np
import pytest

from conftest import GOLDEN_DIR
from oracle import vote_oracle as vo

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("copies,nb", [(1, 3), (1, 4), (1, 7), (1, 8), (12, 8), (12, 3), (90, 5), (300, 4)])
def test_lists_and_groups(cuda, copies, nb):
    import torch
    from pyebsdindex_gb300 import tripletvote as tv
    lib, params, ins, _ = vo.load_case(os.path.join(GOLDEN_DIR, "vote_fcc_syn.npz"))
    lib = dict(lib)
    keep = max(1, 7000 // copies)
    for k in ("trip_angles", "trip_familyid"):
        lib[k] = np.tile(lib[k][:keep], (copies, 1))
    n = 33
    norms, inten = ins["norms"][:n, :nb].copy(), ins["inten"][:n, :nb].copy()
    inten[5, nb // 2] = 0.0
    bi = tv.BandIndexer(lib=lib, angTol=params["angTol"], nband_earlyexit=params["nband_earlyexit"],
                        simpleqweights=params["simpleqweights"], high_fidelity=True)
    got = bi.bandindex_device(torch.from_numpy(norms).cuda(), torch.from_numpy(inten).cuda(), intermediates=True)
    got = {k: v.cpu().numpy() for k, v in got.items()}
    want, mid = vo.bandindex(lib, params, norms, inten)
    want = dict(zip(("quat", "fit", "cm", "polematch", "nmatch", "ij", "acc_correct", "bandfit"), want))
    same = np.ones(n, bool)
    for k, v in (("nmatch", want["nmatch"]), ("polematch", want["polematch"]), ("accn", mid["accn"])):
        same &= (got[k].reshape(n, -1) == np.asarray(v).reshape(n, -1)).all(1)
    assert same.mean() >= 0.9
    np.testing.assert_allclose(got["accw"][same], mid["accw"][same], rtol=1e-5, atol=1e-4)
