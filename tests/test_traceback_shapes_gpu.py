"""Tracebacks over the row blocks of the kernel (4 rows a lane, 128 a warp,
several warps a record, several rounds of warps): coordinates, CIGARs and
scores equal the oracle's, ties included."""
import numpy as np
import pytest

import oracle
from swhybrid_b200 import capi, param, synth

pytestmark = pytest.mark.gpu
M = param.blosum62()
KEYS = ("score", "q_begin", "q_end", "d_begin", "d_end", "cigar")


@pytest.mark.parametrize("qlen", [1, 4, 127, 128, 129, 600, 2049, 4096, 4300])
@pytest.mark.parametrize("gap_open,gap_extend", [(10, 2), (2, 1)])
def test_traceback_equals_oracle(qlen, gap_open, gap_extend):
    rng = np.random.default_rng(qlen)
    q = synth.residues(rng, qlen)
    recs = [synth.residues(rng, n) for n in (1, 31, 33, 300)]
    recs += [synth.mutate(rng, q, 0.2, 0.05) if qlen > 1 else q, q]
    rep = np.concatenate([q, q])                     # the same alignment twice: the first wins
    if qlen <= 2049:
        recs += [rep, np.concatenate([q[:qlen // 2], synth.residues(rng, 40), q[qlen // 2:]])]
    off = np.zeros(len(recs) + 1, dtype=np.uint64)
    off[1:] = np.cumsum([len(r) for r in recs])
    with capi.Context(0, capi.default_params(gap_open=gap_open, gap_extend=gap_extend)) as c:
        c.load_db(np.concatenate(recs).astype(np.uint8), off)
        got = c.traceback(q, list(range(len(recs))))
    for i, (r, al) in enumerate(zip(recs, got)):
        want = oracle.traceback(q, r, M, gap_open + gap_extend, gap_extend)
        assert {k: al[k] for k in KEYS} == {k: want[k] for k in KEYS}, f"record {i} ({len(r)})"


def test_tie_across_row_rounds():
    """The same score ends late in the first 4,096 rows and early in the next
    ones: the smaller record position wins."""
    w, h = param.encode("W" * 8), param.encode("H" * 11)      # 88 each
    q = param.encode("A" * 4600).astype(np.uint8)
    q[100:108] = w
    q[4200:4211] = h
    gap = param.encode("P" * 30)
    recs = [np.concatenate(x).astype(np.uint8) for x in ((gap, h, gap, w, gap), (gap, w, gap, h))]
    off = np.zeros(3, dtype=np.uint64)
    off[1:] = np.cumsum([len(r) for r in recs])
    with capi.Context(0) as c:
        c.load_db(np.concatenate(recs), off)
        got = c.traceback(q, [0, 1])
    for r, al in zip(recs, got):
        want = oracle.traceback(q, r, M, 12, 2)
        assert {k: al[k] for k in KEYS} == {k: want[k] for k in KEYS}
