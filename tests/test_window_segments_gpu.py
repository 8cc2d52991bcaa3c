"""Windows of a long pair in bulk launches over two row segments.  A shape
override makes the windows certain, a query longer than one launch's profile the
segments: the boundary rows of window copies last from one launch to the next,
scores merge by maximum over windows and segments, and a record whose lanes may
have wrapped in several of them is listed once."""
import numpy as np
import pytest

import oracle
from swhybrid_b200 import capi, param, synth

pytestmark = pytest.mark.gpu
M = param.blosum62()
OPEN, EXTEND = 10, 100          # dear gaps: alignments span little beyond the query


def test_windows_over_row_segments():
    rng = np.random.default_rng(19)
    w = param.encode("W" * 4000).astype(np.uint8)
    # 8,192 rows in the first segment: it scores 2,892 of the 4,000 Ws (31,812 of
    # 44,000), past the 16-bit range like the second
    q = np.concatenate([synth.residues(rng, 5300), w]).astype(np.uint8)
    lens = np.concatenate([rng.integers(350, 451, size=68_000), [40_000, 39_000, 12_000]])
    lens = lens[rng.permutation(len(lens))]
    db = synth.db_from_lengths(rng, lens)
    at = [int(np.nonzero(lens == n)[0][0]) for n in (40_000, 39_000, 12_000)]
    for i, start in ((0, 3_000), (0, 18_000), (1, 35_000)):
        o = int(db.offsets[at[i]]) + start
        if i == 0:
            db.residues[o:o + 4000] = w
        else:                                  # a homolog of rows on both sides of the cut
            db.residues[o:o + 2500] = np.where(rng.random(2500) < 0.9, q[2500:5000],
                                               db.residues[o:o + 2500])
    o = int(db.offsets[at[2]])
    db.residues[o + 6000:o + 7500] = w[:1500]
    with capi.Context(0, capi.default_params(gap_open=OPEN, gap_extend=EXTEND,
                                             reference_cap=False)) as c:
        c.load_db(db.residues, db.offsets)
        c.set_kernel_config((32, 64, 32, 64, 0))
        hits, scores = c.search(q, want_scores=True)
        st = c.run_stats()
        # the same shape for the whole DB without windows or a split
        c.set_kernel_config((32, 64, 32, 64, 1 << 29))
        plain_hits, plain = c.search(q, want_scores=True)
        whole = c.run_stats()
    assert st.used.cutover == 0 and st.rescored == 1
    # the windows, a launch per segment, the re-score and two top-k rounds
    assert (st.launches, whole.launches) == (6, 5)
    np.testing.assert_array_equal(scores, plain)
    assert hits == plain_hits and hits[0] == (44_000, at[0])
    pick = np.concatenate([at, rng.choice(db.n, size=40, replace=False)])
    sub = db.subset(pick)
    np.testing.assert_array_equal(
        scores[pick], oracle.search(q, sub.residues, sub.offsets, M, OPEN + EXTEND, EXTEND, mode=0))
