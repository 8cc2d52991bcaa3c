"""A cut-over in a caller's table is for DBs whose groups get at least that many
columns each: on a smaller one the bulk launch would end on pairs just below it."""
import numpy as np
import pytest

import oracle
from swhybrid_b200 import capi, param, synth

pytestmark = pytest.mark.gpu
M = param.blosum62()


@pytest.mark.parametrize("cutover,applies", [(4096, False), (120, True)])
def test_cutover_beyond_a_groups_share(cutover, applies):
    rng = np.random.default_rng(7)
    # 4x40: 96 groups an SM, about 150 columns each
    lens = np.concatenate([rng.integers(80, 111, size=46_000), [9000, 8000, 4000, 3900, 140, 140]])
    db = synth.db_from_lengths(rng, lens[rng.permutation(len(lens))])
    q = synth.residues(rng, 1434)
    with capi.Context(0) as c:
        c.load_db(db.residues, db.offsets)
        c.set_tuning([(100_000, (4, 40, 4, 40, cutover))])
        for _ in range(2):
            hits, scores = c.search(q, want_scores=True)
        st = c.run_stats()
        c.set_tuning([(100_000, (4, 40, 4, 40, 0))])
        for _ in range(2):
            c.search(q)
        free = c.run_stats()
    np.testing.assert_array_equal(scores, oracle.search(q, db.residues, db.offsets, M, 12, 2))
    if applies:
        assert st.used.cutover == cutover
    else:       # as without one; with it, 4,000 columns follow one another in nine passes
        assert st.used.cutover == free.used.cutover and st.kernel_ms < 1.5 * free.kernel_ms
