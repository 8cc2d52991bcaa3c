"""sw_score_noalloc over its row counts, passes, windows and profile forms:
every score equals the oracle's exact one."""
import numpy as np
import pytest

import oracle
from swhybrid_b200 import capi, param, synth

pytestmark = pytest.mark.gpu
M = param.blosum62()


@pytest.mark.parametrize("qlen,n,longs,gap_open,gap_extend", [
    (1, 40, (), 10, 2),
    (128, 300, (8192,), 10, 2),             # 4 rows a lane, one window record
    (129, 300, (8192, 5000, 1), 10, 2),     # 8 rows
    (384, 300, (8192, 8191), 10, 2),        # 12
    (385, 300, (8000,) * 9, 11, 1),         # 16
    (513, 200, (6000,), 10, 2),             # 24, byte profile
    (1024, 200, (8192,), 10, 2),            # 32
    (1025, 100, (8192,), 10, 40),           # 48, windows of a long query
    (2048, 100, (8192,), 10, 2),            # 64
    (2049, 100, (8192,) * 3, 10, 2),        # two passes
    (4500, 60, (3000,), 0, 0),              # three passes, free extension: no windows
    (9000, 20, (300,), 10, 2),              # scores looked up in the matrix
])
def test_noalloc_equals_oracle(qlen, n, longs, gap_open, gap_extend):
    import torch
    rng = np.random.default_rng(qlen)
    q = synth.residues(rng, qlen)
    recs = [synth.residues(rng, int(x)) for x in rng.integers(0, 500, size=n)]
    for x in longs:                          # homologs all along the long records
        r = synth.residues(rng, x)
        for at in range(0, x - qlen, max(3 * qlen, 700)):
            r[at:at + qlen] = np.where(rng.random(qlen) < 0.8, q, r[at:at + qlen])
        recs.insert(int(rng.integers(0, len(recs) + 1)), r)
    off = np.zeros(len(recs) + 1, dtype=np.uint64)
    off[1:] = np.cumsum([len(r) for r in recs])
    res = np.concatenate(recs).astype(np.uint8)
    dev = torch.device("cuda:0")
    d_res, d_q = torch.from_numpy(res).to(dev), torch.from_numpy(q).to(dev)
    d_off = torch.from_numpy(off.astype(np.int64)).to(dev)
    d_out = torch.full((len(recs),), -7, dtype=torch.int32, device=dev)
    p = capi.default_params(gap_open=gap_open, gap_extend=gap_extend, reference_cap=False)
    assert capi.score_noalloc(0, p, d_q.data_ptr(), qlen, d_res.data_ptr(), d_off.data_ptr(),
                              len(recs), d_out.data_ptr()) == capi.SW_OK
    want = oracle.search(q, res, off, M, gap_open + gap_extend, gap_extend, mode=0)
    np.testing.assert_array_equal(d_out.cpu().numpy(), want)
