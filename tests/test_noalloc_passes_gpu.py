"""sw_score_noalloc at the tallest byte profile (8,192 query rows in four passes)
and one row above, where scores are looked up, and in several passes over windows:
boundary-row slices as long as a window, fewer slices than warps."""
import numpy as np
import pytest

import oracle
from swhybrid_b200 import capi, param, synth

pytestmark = pytest.mark.gpu
M = param.blosum62()


@pytest.mark.parametrize("qlen,lens,gap_open,gap_extend", [
    (8192, (1, 300, 2500, 8192), 10, 2),
    (8193, (1, 300, 2500, 8192), 10, 2),
    (2049, (8192,) * 12 + (400,) * 40, 10, 40),     # windows of about 3,300 columns
    (2100, (8192, 8191, 8190, 6000, 50), 10, 40),
    (4097, (8192,) * 6 + (7000, 90), 30, 200),      # three passes
])
def test_noalloc_passes(qlen, lens, gap_open, gap_extend):
    import torch
    rng = np.random.default_rng(qlen + len(lens))
    q = synth.residues(rng, qlen)
    db = synth.db_from_lengths(rng, np.array(lens))
    for i in range(db.n):                    # the query or a part of it, at either end or between
        n = int(db.offsets[i + 1] - db.offsets[i])
        part = q[:min(n, qlen)] if i % 2 else q[max(qlen - n, 0):]
        at = int(db.offsets[i]) + (0, n - len(part), (n - len(part)) // 2)[i % 3]
        keep = rng.random(len(part)) < 0.8
        db.residues[at:at + len(part)] = np.where(keep, part, db.residues[at:at + len(part)])
    dev = torch.device("cuda:0")
    d_res, d_q = torch.from_numpy(db.residues).to(dev), torch.from_numpy(q).to(dev)
    d_off = torch.from_numpy(db.offsets.astype(np.int64)).to(dev)
    d_out = torch.full((db.n,), -7, dtype=torch.int32, device=dev)
    p = capi.default_params(gap_open=gap_open, gap_extend=gap_extend, reference_cap=False)
    assert capi.score_noalloc(0, p, d_q.data_ptr(), qlen, d_res.data_ptr(), d_off.data_ptr(), db.n,
                              d_out.data_ptr()) == capi.SW_OK
    want = oracle.search(q, db.residues, db.offsets, M, gap_open + gap_extend, gap_extend, mode=0)
    np.testing.assert_array_equal(d_out.cpu().numpy(), want)
