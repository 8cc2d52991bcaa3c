"""A shape override on a DB with a long tail and a few records far longer: the SMs
are divided so that the long and the bulk launch of the split end together."""
import numpy as np
import pytest

import oracle
from swhybrid_b200 import capi, param, synth

pytestmark = pytest.mark.gpu
M = param.blosum62()


@pytest.mark.parametrize("shape", [(4, 40), (8, 40), (8, 16)])
def test_long_and_bulk_launch_end_together(shape):
    db = synth.full_db(7, 60_000, 20)
    q = synth.query(8, 500)
    with capi.Context(0) as c:
        c.load_db(db.residues, db.offsets)
        c.set_kernel_config((*shape, *shape, 0))
        for _ in range(3):
            hits, scores = c.search(q, want_scores=True)
        st = c.run_stats()
    assert st.used.cutover >= 1024 and st.long_ms > 0      # a split, no windows
    assert st.bulk_ms < 1.5 * st.long_ms and st.long_ms < 2 * st.bulk_ms, (st.long_ms, st.bulk_ms)
    pick = np.concatenate([np.argsort(-db.lengths())[:3],
                           np.random.default_rng(3).choice(db.n, size=300, replace=False)])
    sub = db.subset(pick)
    np.testing.assert_array_equal(scores[pick], oracle.search(q, sub.residues, sub.offsets, M, 12, 2))
