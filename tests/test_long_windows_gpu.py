"""Short queries against a few long records: the long-pair kernel scores windows
of the longest records (a pipeline's columns are serial).  Scores must equal
the oracle's with gaps as long as the scores can pay for, for records a window
edge either way, and a lane that wraps in several windows is re-scored once."""
import numpy as np
import pytest

import oracle
from swhybrid_b200 import capi, param, synth
from test_windows_gpu import gapped_copies, with_long

pytestmark = pytest.mark.gpu
M = param.blosum62()


def windows_ran(st):
    # windows, long-pair, bulk, re-score and one top-k round; without windows the
    # long-pair launch ends long after the bulk one (no join), which makes four
    return st.used.cutover > 0 and st.used.long_group_width == 32 and st.launches >= 5


@pytest.mark.parametrize("qlen,gap_open,gap_extend,lengths", [
    (40, 10, 2, (30_001, 30_000, 8192, 8191)),
    (120, 10, 2, (20_000, 20_001, 5003)),
    (120, 11, 1, (35_000, 12_007)),         # spans up to 1,400 columns
    (31, 0, 3, (9_999,)),                   # one long record, paired with a short one
])
def test_windows_in_the_long_pair_kernel(qlen, gap_open, gap_extend, lengths):
    rng = np.random.default_rng(3 * qlen + gap_open)
    q = param.encode("W" * (qlen // 2) + "Y" * (qlen - qlen // 2)).astype(np.uint8)
    pays = (7 * (qlen // 2) - gap_open) // gap_extend
    longs = [gapped_copies(rng, q, n, 1, pays + 2, 3 * qlen) for n in lengths]
    res, off = with_long(rng, 1500, 20, 400, longs)
    want = oracle.search(q, res, off, M, gap_open + gap_extend, gap_extend, mode=0)
    with capi.Context(0, capi.default_params(gap_open=gap_open, gap_extend=gap_extend)) as c:
        c.load_db(res, off)
        for _ in range(2):
            hits, scores = c.search(q, want_scores=True)
            assert windows_ran(c.run_stats())
            np.testing.assert_array_equal(scores, want)
            ws, wi = oracle.topk(want, 10)
            assert hits == list(zip(ws.tolist(), wi.tolist()))


def test_lane_that_wraps_in_several_long_windows():
    rng = np.random.default_rng(5)
    m = M.copy()
    w = int(param.encode("W")[0])
    m[w, w] = 90
    q = param.encode("W" * 370).astype(np.uint8)
    rec = np.concatenate([synth.residues(rng, 5000), q, synth.residues(rng, 14_000), q,
                          synth.residues(rng, 17_000)]).astype(np.uint8)
    res, off = with_long(rng, 1500, 300, 500, [rec])
    with capi.Context(0, capi.default_params(gap_open=10, gap_extend=20, matrix=m)) as c:
        c.load_db(res, off)
        hits, scores = c.search(q, want_scores=True)
        st = c.run_stats()
    assert windows_ran(st) and st.rescored == 1
    np.testing.assert_array_equal(scores, oracle.search(q, res, off, m, 30, 20, mode=0))
    assert scores[-1] >= 33_000
