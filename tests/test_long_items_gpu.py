"""Long pairs of a batch (and of served requests) scored beside the
paired-query launches: records far longer than a group's share, queries of
every row count and pass count of those items; scores equal the oracle's and
the plain search's."""
import numpy as np
import pytest

import oracle
from swhybrid_b200 import capi, param, synth

pytestmark = pytest.mark.gpu
M = param.blosum62()


@pytest.fixture(scope="module")
def case():
    rng = np.random.default_rng(41)
    lens = np.concatenate([rng.integers(20, 400, size=1500), [9000, 8999, 7000, 5000, 3001, 3000, 2999]])
    lens = lens[rng.permutation(len(lens))]
    db = synth.db_from_lengths(rng, lens)
    qlens = [1, 31, 128, 129, 700, 2048, 2049, 4096, 4097, 6000]
    queries = [synth.residues(rng, n) for n in qlens]
    for i in np.argsort(-lens)[:3]:                   # homologs inside the longest records
        q = queries[4 + int(i) % 3]
        at = int(db.offsets[i]) + 1500
        db.residues[at:at + len(q)] = np.where(rng.random(len(q)) < 0.85, q,
                                               db.residues[at:at + len(q)])
    return db, queries


@pytest.mark.parametrize("gap_open,gap_extend,picks", [
    (10, 2, range(10)), (11, 1, (0, 3, 5)), (4, 3, (2, 6)), (10, 2, (9,)), (10, 2, (0, 1)),
])
def test_batch_with_long_records(case, gap_open, gap_extend, picks):
    db, queries = case
    qs = [queries[i] for i in picks]
    with capi.Context(0, capi.default_params(gap_open=gap_open, gap_extend=gap_extend)) as c:
        c.load_db(db.residues, db.offsets)
        for _ in range(2):                            # captured, then replayed
            hits, scores = c.search_batch(qs, want_scores=True)
        plain = [c.search(q) for q in qs]
    for q, sc, h, p in zip(qs, scores, hits, plain):
        want = oracle.search(q, db.residues, db.offsets, M, gap_open + gap_extend, gap_extend, mode=0)
        np.testing.assert_array_equal(sc, want, err_msg=f"query of {len(q)}")
        assert h == p[0]


def test_saturated_long_record_in_a_batch():
    rng = np.random.default_rng(42)
    w = param.encode("W" * 3100).astype(np.uint8)
    rec = np.concatenate([synth.residues(rng, 3000), w, synth.residues(rng, 4000)]).astype(np.uint8)
    db = synth.db_from_lengths(rng, rng.integers(50, 300, size=800))
    res = np.concatenate([db.residues, rec]).astype(np.uint8)
    off = np.concatenate([db.offsets, [len(res)]]).astype(np.uint64)
    qs = [w, synth.residues(rng, 100)]
    with capi.Context(0) as c:
        c.load_db(res, off)
        hits, scores = c.search_batch(qs, want_scores=True)
        assert c.run_stats().rescored == 1
    assert scores[0][-1] == oracle.gotoh(w, rec, M) >= 34_000
    np.testing.assert_array_equal(scores[1], oracle.search(qs[1], res, off, M, 12, 2))


@pytest.mark.parametrize("chunks", [1, 4])
def test_served_requests_with_long_records(case, chunks):
    """Requests score the long pairs in their first round, whatever else is in
    flight; each list equals the plain search's."""
    db, queries = case
    with capi.Context(0) as c:
        c.load_db(db.residues, db.offsets)
        plain = [c.search(q)[0] for q in queries]
        c.serve_start(chunks=chunks, max_active=6)
        got, sent = {}, 0
        while len(got) < 2 * len(queries):
            if sent < 2 * len(queries):
                c.serve_submit(sent, queries[sent % len(queries)])
                sent += 1
            for r in c.serve_poll(timeout_ms=0 if sent < 2 * len(queries) else 5000):
                assert r["status"] == 0
                got[r["id"]] = r["hits"]
        c.serve_stop()
    for i, h in got.items():
        assert h == plain[i % len(queries)], f"request {i}"
