"""The first pass has a narrow cell for matrices whose entries lie in
[-(open + extend), 127 - (open + extend)] and a wide one for the rest.  Matrices
at, just inside and just outside either end must give the oracle's scores in
the plain search, its long-pair launch and the paired and stacked batch
launches."""
import numpy as np
import pytest

import oracle
from swhybrid_b200 import capi, param, synth

pytestmark = pytest.mark.gpu
ALPHA = param.ALPHABET


def edge_matrix(seed, lo, hi):
    """Symmetric, both ends taken on and off the diagonal; mostly low entries,
    so that scores stay below the 32-bit pass's limit now and then."""
    rng = np.random.default_rng(seed)
    r = rng.integers(lo, max(lo // 2, lo + 1) + 1, size=(23, 23))
    r = np.triu(r) + np.triu(r, 1).T
    r[np.arange(23), np.arange(23)] = rng.integers(1, 9, size=23)
    r[3, 3] = hi
    r[5, 8] = r[8, 5] = hi
    r[2, 6] = r[6, 2] = lo
    lines = ["   " + " ".join(ALPHA)]
    lines += [ALPHA[i] + " " + " ".join(str(int(v)) for v in r[i]) for i in range(23)]
    return capi.parse_matrix("\n".join(lines) + "\n")


@pytest.mark.parametrize("go,ge", [(10, 2), (11, 1), (7, 3), (0, 1)])
@pytest.mark.parametrize("below,above", [(0, 0), (1, 0), (0, 1)])
def test_matrix_edges_of_the_narrow_cell(go, ge, below, above):
    q_cost = go + ge
    m = edge_matrix(go * 16 + ge, -q_cost - below, 127 - q_cost + above)
    rng = np.random.default_rng(17 + go)
    db = synth.small_db(23 + ge, 700)
    long_rec = synth.residues(rng, 5003).astype(np.uint8)
    off = np.concatenate([db.offsets, [db.offsets[-1] + np.uint64(len(long_rec))]]).astype(np.uint64)
    res = np.concatenate([db.residues, long_rec]).astype(np.uint8)
    qs = [synth.residues(rng, L) for L in (37, 300, 1100)]
    want = [oracle.search(q, res, off, m, q_cost, ge, mode=0) for q in qs]
    params = capi.default_params(gap_open=go, gap_extend=ge, matrix=m, reference_cap=False)
    with capi.Context(0, params) as c:
        c.load_db(res, off)
        for q, w in zip(qs, want):
            np.testing.assert_array_equal(c.search(q, want_scores=True)[1], w)
        c.set_kernel_config((16, 8, 32, 16, 2000))          # one record to the long-pair kernel
        for q, w in zip(qs, want):
            np.testing.assert_array_equal(c.search(q, want_scores=True)[1], w)
            assert c.run_stats().used.cutover > 0
        _, b = c.search_batch(qs, want_scores=True)
        for qi, w in enumerate(want):
            np.testing.assert_array_equal(b[qi], w)
