"""Long-pair kernel, the row counts between its older ones: query lengths at
the edges of one and several passes must give the oracle's scores."""
import numpy as np
import pytest

import oracle
from swhybrid_b200 import capi, param, synth

pytestmark = pytest.mark.gpu
M = param.blosum62()


@pytest.mark.parametrize("rows", [4, 6, 12, 20])
@pytest.mark.parametrize("go,ge", [(10, 2), (11, 1), (8, 2)])
def test_long_rows_at_pass_edges(rows, go, ge):
    rng = np.random.default_rng(rows + go)
    db = synth.db_from_lengths(rng, np.concatenate([rng.integers(20, 300, size=300),
                                                    [2500, 2501, 3999, 4000, 4001]]))
    with capi.Context(0, capi.default_params(gap_open=go, gap_extend=ge)) as c:
        c.load_db(db.residues, db.offsets)
        c.set_kernel_config((32, rows, 16, 8, 2000))
        for qlen in (32 * rows - 1, 32 * rows, 32 * rows + 1, 96 * rows + 5):
            q = synth.residues(rng, qlen)
            _, scores = c.search(q, want_scores=True)
            u = c.run_stats().used
            assert u.cutover > 0 and u.long_rows_per_thread == rows
            np.testing.assert_array_equal(
                scores, oracle.search(q, db.residues, db.offsets, M, go + ge, ge, mode=0))
