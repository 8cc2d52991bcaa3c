"""Long records in overlapping windows: a plain search cuts the pairs that hold
more columns than an evenly loaded group gets into windows that overlap by the
longest span an alignment of the query can have, and takes the maximum over a
record's windows.  Scores must equal the oracle's wherever an alignment lies,
with gaps as long as the scores can pay for, and a lane that wraps in several
windows is re-scored once."""
import numpy as np
import pytest

import oracle
from swhybrid_b200 import capi, param, synth

pytestmark = pytest.mark.gpu
M = param.blosum62()


def with_long(rng, n, lo, hi, longs):
    lens = np.concatenate([rng.integers(lo, hi + 1, size=n), [len(x) for x in longs]])
    off = np.zeros(len(lens) + 1, dtype=np.uint64)
    off[1:] = np.cumsum(lens)
    short = synth.residues(rng, int(off[n]))
    return np.concatenate([short] + longs).astype(np.uint8), off


def gapped_copies(rng, q, length, gap_lo, gap_hi, every):
    """A record holding both halves of q again and again, `gap` residues of A
    between them (A against a W run never matches)."""
    a = param.encode("A")[0]
    out, h = [], len(q) // 2
    while sum(len(x) for x in out) < length:
        out += [q[:h], np.full(int(rng.integers(gap_lo, gap_hi)), a), q[h:],
                np.full(int(rng.integers(every // 2, every)), a)]
    return np.concatenate(out)[:length].astype(np.uint8)


@pytest.mark.parametrize("qlen,gap_open,gap_extend,lengths", [
    (120, 10, 2, (3001, 8192, 20000)),      # default gaps
    (120, 11, 1, (9000, 15007)),            # spans up to 1,400 columns
    (64, 0, 3, (2500, 2504, 2505, 6000)),   # one window more per few columns
    (31, 5, 4, (1999, 35000)),
])
def test_windowed_records_equal_the_oracle(qlen, gap_open, gap_extend, lengths):
    rng = np.random.default_rng(qlen + gap_open)
    q = param.encode("W" * (qlen // 2) + "Y" * (qlen - qlen // 2)).astype(np.uint8)
    # the longest gap that still pays: half of the alignment's score
    pays = (7 * (qlen // 2) - gap_open) // gap_extend
    longs = [gapped_copies(rng, q, n, 1, pays + 2, 3 * qlen) for n in lengths]
    res, off = with_long(rng, 40_000, 150, 350, longs)
    with capi.Context(0, capi.default_params(gap_open=gap_open, gap_extend=gap_extend)) as c:
        c.load_db(res, off)
        c.set_kernel_config((16, 64, 16, 64, 0))            # ~2,100 columns per group
        hits, scores = c.search(q, want_scores=True)
        st = c.run_stats()
        # windows + first pass + re-score + two top-k rounds, no long-pair split
        assert st.used.cutover == 0 and st.launches == 5
    want = oracle.search(q, res, off, M, gap_open + gap_extend, gap_extend, mode=0)
    np.testing.assert_array_equal(scores, want)
    assert scores[-1] > 11 * (qlen // 2)        # both halves across a gap
    ws, wi = oracle.topk(want, 10)
    assert hits == list(zip(ws.tolist(), wi.tolist()))


@pytest.mark.parametrize("row_segments", [False, True])
def test_saturation_in_overlapping_windows(row_segments):
    """W runs of 370 (90 per cell) in a 40,000-residue record: the lane wraps
    in every window that holds one, and the record is listed for the 32-bit
    pass once, also when the query's rows run as two segments."""
    rng = np.random.default_rng(9)
    m = M.copy()
    w = int(param.encode("W")[0])
    m[w, w] = 90
    q = param.encode("W" * 370).astype(np.uint8)
    rec = np.concatenate([synth.residues(rng, 5000), q, synth.residues(rng, 17_000), q,
                          synth.residues(rng, 17_000)]).astype(np.uint8)
    res, off = with_long(rng, 60_000, 300, 500, [rec])
    with capi.Context(0, capi.default_params(gap_open=10, gap_extend=20, matrix=m)) as c:
        c.load_db(res, off)
        if row_segments:
            c.set_tuning([(1 << 30, (32, 8, 32, 8, 0), ((32, 8, 1), (32, 8, 0)))])
        else:
            c.set_kernel_config((32, 8, 32, 8, 0))
        assert len(c.plan(370)) == (2 if row_segments else 1)
        hits, scores = c.search(q, want_scores=True)
        st = c.run_stats()
    assert st.rescored == 1
    # (with the table the time model may send the one long pair to the
    # long-pair kernel instead)
    assert row_segments or (st.used.cutover == 0 and st.launches == 5)
    top = oracle.gotoh(q, rec, m, 30, 20)
    assert top >= 33_000 and scores[-1] == top and hits[0] == (top, len(off) - 2)
    pick = rng.choice(60_000, size=200, replace=False)
    sub = synth.DB(res, off).subset(pick)
    np.testing.assert_array_equal(scores[pick], oracle.search(q, sub.residues, sub.offsets, m, 30, 20,
                                                              mode=0))
