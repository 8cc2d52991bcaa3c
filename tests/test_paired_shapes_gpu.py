"""Every paired-query kernel shape, batched and served, on an odd number of pairs
(and of records): the groups of a warp claim units side by side, so the last
claim of a chunk reaches past its end.  Scores and hit lists equal the oracle's."""
import numpy as np
import pytest

import oracle
from swhybrid_b200 import capi, param, synth

pytestmark = pytest.mark.gpu
M = param.blosum62()
# (shape, rows of a paired lane: whole passes whose profile fits a block)
SHAPES = [((8, 64), 512), ((8, 64), 1024), ((16, 64), 2048), ((16, 48), 1536), ((16, 32), 2048),
          ((32, 32), 2048)]
QLENS = (7, 64, 375, 700, 1300, 2600)


@pytest.fixture(scope="module")
def case():
    rng = np.random.default_rng(91)
    lens = np.concatenate([rng.integers(1, 300, size=601), [2400, 1700]])    # 603 records, 302 pairs
    db = synth.db_from_lengths(rng, lens[rng.permutation(len(lens))])
    return db, [synth.residues(rng, n) for n in QLENS]


def wanted(db, queries, oe=12, e=2):
    out = []
    for q in queries:
        ws, wi = oracle.topk(oracle.search(q, db.residues, db.offsets, M, oe, e, mode=0), 10)
        out.append(list(zip(ws.tolist(), wi.tolist())))
    return out


@pytest.mark.parametrize("chunks", [1, 3, 301])
@pytest.mark.parametrize("shape,rows", SHAPES)
def test_served_with_every_paired_shape(case, shape, rows, chunks):
    db, queries = case
    db = db.subset(np.arange(db.n - 2 * (chunks == 1)))      # one chunk: 301 pairs
    want = wanted(db, queries)
    with capi.Context(0) as c:
        c.load_db(db.residues, db.offsets)
        c.serve_start(chunks=chunks, max_active=8, pair_shape=shape, pair_rows=rows)
        try:
            for i, q in enumerate(queries):
                assert c.serve_submit(i, q) == 0
            got = {}
            while len(got) < len(queries):
                for r in c.serve_poll(timeout_ms=5000):
                    assert r["status"] == 0
                    got[r["id"]] = r["hits"]
        finally:
            c.serve_stop()
    assert [got[i] for i in range(len(queries))] == want


@pytest.mark.parametrize("gap_open,gap_extend", [(8, 2), (12, 3), (1, 1), (300, 300)])
@pytest.mark.parametrize("shape,rows", SHAPES)
def test_batch_at_run_time_gap_costs(case, shape, rows, gap_open, gap_extend):
    """Gap costs without a kernel of their own, also where the matrix is too wide
    for the plain kernel's narrow cell (1/1) and past any score's reach (300/300)."""
    db, queries = case
    with capi.Context(0, capi.default_params(gap_open=gap_open, gap_extend=gap_extend)) as c:
        c.load_db(db.residues, db.offsets)
        c.set_batch_options(pair_shape=shape, pair_rows=rows)
        hits, scores = c.search_batch(queries, want_scores=True)
    for q, sc, h, w in zip(queries, scores, hits,
                           wanted(db, queries, gap_open + gap_extend, gap_extend)):
        want = oracle.search(q, db.residues, db.offsets, M, gap_open + gap_extend, gap_extend, mode=0)
        np.testing.assert_array_equal(sc, want, err_msg=f"query of {len(q)}")
        assert h == w
