"""sw_score_noalloc with so many records that its long ones are claimed four
neighbours at a time: the last group partly filled, long neighbours of unequal
window counts."""
import numpy as np
import pytest

import oracle
from swhybrid_b200 import capi, param, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [40_000, 40_001, 40_003])
def test_noalloc_many_records(n):
    import torch
    rng = np.random.default_rng(n)
    lens = rng.integers(0, 60, size=n)
    lens[[0, 1, 2, 5, n - 3, n - 2, n - 1]] = [8192, 3000, 700, 8191, 5000, 129, 2600]
    db = synth.db_from_lengths(rng, lens)
    q = synth.residues(rng, 30)
    dev = torch.device("cuda:0")
    d_res, d_q = torch.from_numpy(db.residues.astype(np.uint8)).to(dev), torch.from_numpy(q).to(dev)
    d_off = torch.from_numpy(db.offsets.astype(np.int64)).to(dev)
    d_out = torch.full((n,), -7, dtype=torch.int32, device=dev)
    assert capi.score_noalloc(0, capi.default_params(), d_q.data_ptr(), len(q), d_res.data_ptr(),
                              d_off.data_ptr(), n, d_out.data_ptr()) == capi.SW_OK
    want = oracle.search(q, db.residues, db.offsets, param.blosum62(), 12, 2, mode=0)
    np.testing.assert_array_equal(d_out.cpu().numpy(), want)
