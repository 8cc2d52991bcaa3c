"""A batch replays a captured graph only while the shapes behind it stand: a
shape override or a tuning table set between two batches of the same lengths
gives the stacks of the second one another kernel, grid and row map."""
import numpy as np
import pytest

import oracle
from swhybrid_b200 import capi, param, synth

pytestmark = pytest.mark.gpu
M = param.blosum62()
SHAPES = [(16, 32), (8, 16), (32, 8), (16, 32)]


@pytest.mark.parametrize("setter", ["override", "table"])
def test_batch_after_a_change_of_shape(setter):
    rng = np.random.default_rng(77)
    db = synth.small_db(31, 1200)
    qs = [synth.residues(rng, n) for n in (700, 513, 300, 40)]
    want = [oracle.search(q, db.residues, db.offsets, M, 12, 2, mode=0) for q in qs]
    with capi.Context(0, capi.default_params(top_k=10)) as c:
        c.load_db(db.residues, db.offsets)
        # queries of at least stack_rows: one stack each, shaped by the configuration
        c.set_batch_options(pair_long=False, pair_rows=0, stack_rows=256)
        for T, R in SHAPES:
            cfg = (T, R, T, R, 0)
            if setter == "override":
                c.set_kernel_config(cfg)
            else:
                c.set_tuning([(100_000, cfg)])
            for _ in range(2):                    # captured, then replayed
                hits, scores = c.search_batch(qs, want_scores=True)
                for sc, h, w in zip(scores, hits, want):
                    np.testing.assert_array_equal(sc, w, err_msg=f"{setter} {T}x{R}")
                    ws, wi = oracle.topk(w, 10)
                    assert h == list(zip(ws.tolist(), wi.tolist()))
