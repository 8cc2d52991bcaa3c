"""Stacks of tall queries with the built-in table, no table and a caller's, on a
DB with a few long records: the stacked kernel's shape is chosen for it (a narrow
group would score a long record for most of the batch's time), the scores are the
oracle's."""
import numpy as np
import pytest

import oracle
from swhybrid_b200 import capi, param, synth

pytestmark = pytest.mark.gpu
M = param.blosum62()


@pytest.fixture(scope="module")
def case():
    rng = np.random.default_rng(101)
    lens = np.concatenate([rng.integers(100, 500, size=1500), [20_000, 9_000, 8_999]])
    db = synth.db_from_lengths(rng, lens[rng.permutation(len(lens))])
    qs = [synth.residues(rng, n) for n in (2900, 1450, 1024, 700, 90)]
    want = [oracle.search(q, db.residues, db.offsets, M, 12, 2, mode=0) for q in qs]
    return db, qs, want


@pytest.mark.parametrize("table", ["built-in", "none", "callers"])
@pytest.mark.parametrize("cutover", [0, 4096])
def test_tall_stacks(case, table, cutover):
    db, qs, want = case
    with capi.Context(0, capi.default_params()) as c:
        c.load_db(db.residues, db.offsets)
        c.set_batch_options(pair_rows=0, pair_long=False, stack_rows=1024, cutover=cutover)
        if table == "none":
            c.set_tuning([])
        elif table == "callers":
            c.set_tuning([(100_000, (4, 40, 4, 40, 0))])
        times = []
        for _ in range(3):                        # captured, then replayed
            _, scores = c.search_batch(qs, want_scores=True)
            times.append(c.run_stats().kernel_ms)
            for q, sc, w in zip(qs, scores, want):
                np.testing.assert_array_equal(sc, w, err_msg=f"query of {len(q)}")
    # 2,900 rows are 19 passes of 4x40 over the longest record's 20,000 columns, one
    # after another (380,000 steps, over 170 ms at 1.965 GHz and 900 clocks a step),
    # and three or fewer passes of a wide group
    if table != "callers" and cutover == 0:
        assert min(times) < 100, times
