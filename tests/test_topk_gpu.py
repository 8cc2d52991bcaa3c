"""Hit lists of every length class (repeated maxima up to 128 hits, a sort
above), at record counts around the 4,096-key blocks, with many equal scores:
the oracle's order (score descending, then record ascending)."""
import numpy as np
import pytest

import oracle
from swhybrid_b200 import capi, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [1, 10, 127, 128, 129, 1024])
@pytest.mark.parametrize("n", [1, 3, 4095, 4096, 4097, 12_500])
def test_hit_list(n, k):
    rng = np.random.default_rng(n + k)
    db = synth.db_from_lengths(rng, rng.integers(0, 30, size=n))     # short: few distinct scores
    q = synth.query(k, 40)
    with capi.Context(0, capi.default_params(top_k=k)) as c:
        c.load_db(db.residues, db.offsets)
        hits, scores = c.search(q, want_scores=True)
        batch, _ = c.search_batch([q, q[:7]])
    sc, idx = oracle.topk(scores, k)
    want = [(s, i) for s, i in zip(sc.tolist(), idx.tolist()) if s > 0]
    assert hits == want and batch[0] == want
