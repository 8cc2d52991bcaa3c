"""Performance cases: the calls a user of this package makes, at the sizes they
are made at.

Each case is one pass through a public entry point of ``swhybrid_b200.capi``:

  search     Context.search: one query against the resident DB, host buffers
             (what the reference's GPU worker does per run)
  device     Context.search_device + sync: queries and scores stay on the GPU
  batch      Context.search_batch: many queries in one call (CUDA graph)
  serve      serve_submit / serve_poll: requests through the scheduler
  traceback  Context.traceback: alignments of a search's hits
  noalloc    score_noalloc: the caller's device buffers, no allocation

Databases follow the benchmark's synthetic generator (background residue
frequencies, lognormal lengths, optional planted long records and homologs).
Record lengths depend on the case alone; residues, queries and the records'
order come from the seed.
"""
import math

import numpy as np
import torch

from swhybrid_b200 import capi, param, synth

# Operations of one cell update (substitution add, two gap openings, two
# extensions, and the maxima of H, E, F and the running best).
CELL_OPS = 11


def _case(name, op, **kw):
    c = {"op": op, "records": 20_000, "sigma": 0.6, "long_records": 0, "long_lo": 10_000,
         "long_hi": 35_000, "homologs": 0, "queries": 1, "qlo": 375, "qhi": 375, "top_k": 10,
         "gap_open": 10, "gap_extend": 2, "matrix": "blosum62", "cap": True, "scores": False}
    c.update(kw)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # a short query against a panel of a few hundred proteins: latency only
        _case("search_panel", "search", records=200, qlo=144, qhi=144, scores=True),
        # the small benchmark workload: query 375, 20,000 records, every score
        _case("search_small", "search", scores=True),
        # short and odd-length queries of the benchmark's sweep (144..5,478)
        # against a DB of a fifth of its size, hits only
        _case("search_short", "search", records=114_000, sigma=0.7, long_records=40,
              qlo=144, qhi=144),
        _case("search_medium", "search", records=114_000, sigma=0.7, long_records=40,
              qlo=549, qhi=549),
        # the benchmark's full-size DB (570,200 records, ~202 M residues)
        _case("search_full", "search", records=570_000, sigma=0.7, long_records=200,
              qlo=1434, qhi=1434),
        # the top of the sweep and lengths around it, resident on the GPU:
        # three queries enqueued back to back, every score
        _case("device_long", "device", records=114_000, sigma=0.7, long_records=40, queries=3,
              qlo=2103, qhi=5478, scores=True),
        # other scoring options: gap 11/1, match/mismatch matrix, a long hit
        # list, no 65,535 cap
        _case("search_options", "search", records=40_000, qlo=731, qhi=731, top_k=500,
              gap_open=11, gap_extend=1, matrix="identity", cap=False, scores=True),
        # overflow and long records: 1 % of the records hold 43 % of the
        # residues, 0.5 % are homologs of the query (16-bit lanes overflow)
        _case("search_stress", "search", records=20_000, long_records=200, long_hi=40_000,
              homologs=100, qlo=1900, qhi=1900, scores=True),
        # the batched benchmark: 64 queries of 50..5,000 residues in one call
        _case("batch_64", "batch", records=114_000, sigma=0.7, long_records=40, queries=64,
              qlo=50, qhi=5000),
        # served: 48 requests of 30..8,000 residues queued at once
        _case("serve_48", "serve", records=57_000, sigma=0.7, long_records=20, queries=48,
              qlo=30, qhi=8000),
        # alignments of the ten best hits of an ordinary query
        _case("traceback_hits", "traceback", records=2_000, homologs=10, qlo=1000, qhi=1000),
        # a plug-in that scores its own device buffers without allocating
        _case("noalloc_small", "noalloc", records=10_000, scores=True),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["search", "search", "search", "device", "batch", "serve", "traceback",
                     "noalloc"])
    gaps = rng.choice([(10, 2), (10, 2), (10, 2), (11, 1), (8, 2), (12, 3)])
    kw = dict(sigma=rng.choice([0.6, 0.7]), gap_open=gaps[0], gap_extend=gaps[1],
              matrix=rng.choice(["blosum62", "blosum62", "blosum62", "identity"]),
              cap=rng.random() < 0.8, top_k=rng.choice([1, 10, 10, 10, 50, 500]))
    if op in ("search", "device"):
        n = _log(rng, 150, 150_000)
        q = _log(rng, 40, 5478)
        return _case(None, op, records=n, long_records=rng.choice([0, n // 2000, n // 500]),
                     homologs=rng.choice([0, min(n // 200, 100)]),
                     queries=rng.randint(1, 4) if op == "device" else 1, qlo=q,
                     qhi=max(q, _log(rng, 40, 5478)) if op == "device" else q,
                     scores=op == "device" or rng.random() < 0.4, **kw)
    if op in ("batch", "serve"):
        n = _log(rng, 2_000, 57_000)
        lo = _log(rng, 30, 400)
        return _case(None, op, records=n, long_records=rng.choice([0, n // 2850]),
                     queries=rng.randint(2, 64), qlo=lo,
                     qhi=_log(rng, 2 * lo, 5000 if op == "batch" else 8000), **kw)
    if op == "traceback":
        q = _log(rng, 60, 3000)
        return _case(None, op, records=2_000, homologs=rng.randint(1, 50), qlo=q, qhi=q, **kw)
    q = _log(rng, 40, 1500)
    return _case(None, op, records=_log(rng, 100, 10_000), qlo=q, qhi=q, scores=True, **kw)


def _rng(case, what):
    return np.random.default_rng([what, case["records"], case["long_records"], case["qlo"]])


def _query_lengths(case):
    """Lengths spread over the logarithm of the case's range."""
    n = case["queries"]
    if n == 1:
        return [case["qlo"]]
    return [int(x) for x in np.rint(np.geomspace(case["qlo"], case["qhi"], n))]


def _db_lengths(case):
    rng = _rng(case, 1)
    hi = 5000 if case["sigma"] < 0.65 else 35_000
    lens = synth.lognormal_lengths(rng, case["records"], 5.6, case["sigma"], 20, hi)
    if case["op"] == "noalloc":
        lens = np.minimum(lens, 8192)
    if case["long_records"]:
        lens = np.concatenate([lens, rng.integers(case["long_lo"], case["long_hi"] + 1,
                                                  size=case["long_records"])])
    return lens


def _mutated(rng, seq):
    """A homolog: substitutions at 10..30 %, indels at 2 %."""
    s = seq.copy()
    sub = rng.random(len(s)) < rng.uniform(0.10, 0.30)
    s[sub] = synth.residues(rng, int(sub.sum()))
    s = s[rng.random(len(s)) >= 0.01]
    at = np.nonzero(rng.random(len(s)) < 0.01)[0]
    return np.insert(s, at, synth.residues(rng, len(at)))


def _inputs(case, seed):
    """Queries, and the records as codes back to back with offsets."""
    rng = np.random.default_rng([2, seed])
    lens = _db_lengths(case)
    lens = lens[rng.permutation(len(lens))]
    queries = [synth.residues(rng, n) for n in _query_lengths(case)]
    queries = [queries[i] for i in rng.permutation(len(queries))]
    planted = np.zeros(0, dtype=np.int64)
    extra = {}
    if case["homologs"]:
        planted = np.sort(rng.choice(len(lens), size=case["homologs"], replace=False))
        for j, i in enumerate(planted):
            extra[int(i)] = _mutated(rng, queries[j % len(queries)])
            lens[i] = len(extra[int(i)])
    off = np.zeros(len(lens) + 1, dtype=np.uint64)
    off[1:] = np.cumsum(lens)
    res = synth.residues(rng, int(off[-1]))
    for i, s in extra.items():
        res[int(off[i]):int(off[i]) + len(s)] = s
    return queries, res, off, planted


def _matrix(case):
    if case["matrix"] == "blosum62":
        return np.array(param.blosum62(), dtype=np.int64).reshape(32, 32)
    m = np.zeros((32, 32), dtype=np.int64)      # +5 match, -4 mismatch
    m[:23, :23] = -4
    m[np.arange(23), np.arange(23)] = 5
    return m


def _params(case):
    return capi.default_params(gap_open=case["gap_open"], gap_extend=case["gap_extend"],
                               top_k=case["top_k"], matrix=_matrix(case),
                               reference_cap=case["cap"])


def prepare(case, seed):
    queries, res, off, planted = _inputs(case, seed)
    p = _params(case)
    s = {"case": case, "queries": queries, "params": p}
    if case["op"] == "noalloc":
        s["d_res"] = torch.from_numpy(res).cuda()
        s["d_off"] = torch.from_numpy(off.astype(np.int64)).cuda()
        s["d_query"] = torch.from_numpy(queries[0]).cuda()
        s["d_scores"] = torch.zeros(len(off) - 1, dtype=torch.int32, device="cuda")
        return s
    ctx = capi.Context(0, p)
    ctx.load_db(res, off)
    s["ctx"] = ctx
    if case["op"] == "device":
        s["d_queries"] = [torch.from_numpy(q).cuda() for q in queries]
        s["d_scores"] = torch.zeros(len(queries), len(off) - 1, dtype=torch.int32, device="cuda")
    elif case["op"] == "serve":
        ctx.serve_start()
    elif case["op"] == "traceback":
        s["records"] = planted
    torch.cuda.synchronize()
    return s


def _hit_table(lists, k):
    """Hit lists as one array [query][hit][score, record], rows of zeros after the last."""
    t = np.zeros((len(lists), k, 2), dtype=np.int64)
    for i, h in enumerate(lists):
        if h:
            t[i, :len(h)] = h
    return t


def run(s):
    case = s["case"]
    op, k = case["op"], case["top_k"]
    if op == "search":
        hits, scores = s["ctx"].search(s["queries"][0], want_scores=case["scores"])
        out = {"hits": _hit_table([hits], k)}
        if scores is not None:
            out["scores"] = scores
        return out
    if op == "device":
        for q, sc in zip(s["d_queries"], s["d_scores"]):
            s["ctx"].search_device(q.data_ptr(), q.numel(), sc.data_ptr())
        s["ctx"].sync()
        return {"scores": s["d_scores"]}
    if op == "batch":
        hits, _ = s["ctx"].search_batch(s["queries"])
        return {"hits": _hit_table(hits, k)}
    if op == "serve":
        ctx, n = s["ctx"], len(s["queries"])
        for i, q in enumerate(s["queries"]):
            ctx.serve_submit(i, q)
        lists, left = [None] * n, n
        while left:
            for r in ctx.serve_poll(max_results=n, timeout_ms=10_000):
                if r["status"] != capi.SW_OK:
                    raise RuntimeError("request %d: status %d" % (r["id"], r["status"]))
                lists[r["id"]] = r["hits"]
                left -= 1
        return {"hits": _hit_table(lists, k)}
    if op == "traceback":
        al = s["ctx"].traceback(s["queries"][0], s["records"])
        fields = ("index", "score", "q_begin", "q_end", "d_begin", "d_end", "matches")
        cigars = np.zeros((len(al), 4 * len(s["queries"][0]) + 64), dtype=np.uint8)
        for i, a in enumerate(al):
            cigars[i, :len(a["cigar"])] = np.frombuffer(a["cigar"].encode(), dtype=np.uint8)
        return {"ends": np.array([[a[f] for f in fields] for a in al], dtype=np.int64),
                "cigars": cigars}
    st = capi.score_noalloc(0, s["params"], s["d_query"].data_ptr(), s["d_query"].numel(),
                            s["d_res"].data_ptr(), s["d_off"].data_ptr(),
                            s["d_scores"].numel(), s["d_scores"].data_ptr())
    if st != capi.SW_OK:
        raise RuntimeError("score_noalloc: status %d" % st)
    return {"scores": s["d_scores"]}


def _cells(case):
    q = sum(_query_lengths(case))
    if case["op"] == "traceback":       # the records aligned are homologs of the query
        return q * q * case["homologs"]
    return q * int(_db_lengths(case).sum())


def work(case):
    """The residues read once per call (not per query), the queries, and the
    scores or hits; CELL_OPS integer operations per cell."""
    n = case["records"] + case["long_records"]
    q = _query_lengths(case)
    if case["op"] == "traceback":
        res, out = q[0] * case["homologs"], 48 * case["homologs"]
    else:
        res = int(_db_lengths(case).sum())
        out = (4 * n if case["scores"] else 16 * case["top_k"]) * len(q)
    return {"bytes": res + sum(q) + out, "flops": CELL_OPS * _cells(case)}


def _exact_scores(query, res, off, matrix, gap_open, gap_extend):
    """Smith-Waterman with affine gaps in 64-bit integers: records side by
    side, one anti-diagonal of every record's matrix at a time."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    lens = np.diff(off.astype(np.int64))
    order = np.argsort(-lens, kind="stable")
    mat = torch.as_tensor(matrix, dtype=torch.int64, device=dev).clone()
    mat[24:, :] = 0
    mat[:, 24:] = 0
    rows = mat[torch.as_tensor(query.astype(np.int64), device=dev)]          # [q, 32]
    m = len(query)
    out = np.zeros(len(lens), dtype=np.int64)
    i = 0
    while i < len(order):
        part = order[i:i + 4096]
        part = part[lens[part] * 2 >= lens[part[0]]]      # similar lengths together
        i += len(part)
        width = int(lens[part[0]])
        if width == 0:
            continue
        cols = np.full((len(part), width), 24, dtype=np.int64)
        for r, rec in enumerate(part):
            cols[r, :lens[rec]] = res[int(off[rec]):int(off[rec + 1])]
        # residues padded so that row j's column on anti-diagonal d is d - j
        pad = torch.full((len(part), width + 2 * m), 24, dtype=torch.int64, device=dev)
        pad[:, m:m + width] = torch.as_tensor(cols, device=dev)
        low = -(1 << 40)
        shape = (len(part), m)
        h1 = torch.zeros(shape, dtype=torch.int64, device=dev)     # H on diagonal d - 1
        h2 = torch.zeros_like(h1)                                  # H on diagonal d - 2
        e = torch.full(shape, low, dtype=torch.int64, device=dev)
        f = torch.full(shape, low, dtype=torch.int64, device=dev)
        best = torch.zeros(len(part), dtype=torch.int64, device=dev)
        j = torch.arange(m, device=dev)
        zero = torch.zeros(len(part), 1, dtype=torch.int64, device=dev)
        none = torch.full((len(part), 1), low, dtype=torch.int64, device=dev)
        for d in range(width + m - 1):
            c = d - j
            inside = ((c >= 0) & (c < width)).unsqueeze(0)
            score = rows[j.unsqueeze(0), pad[:, d + m - j]]
            e = torch.maximum(e - gap_extend, h1 - (gap_open + gap_extend))
            up_h = torch.cat([zero, h1[:, :-1]], 1)
            up_f = torch.cat([none, f[:, :-1]], 1)
            f = torch.maximum(up_f - gap_extend, up_h - (gap_open + gap_extend))
            diag = torch.cat([zero, h2[:, :-1]], 1)
            h = torch.maximum(torch.maximum(diag + score, e), f).clamp_(min=0)
            h = torch.where(inside, h, torch.zeros_like(h))
            e = torch.where(inside, e, torch.full_like(e, low))
            f = torch.where(inside, f, torch.full_like(f, low))
            best = torch.maximum(best, h.amax(1))
            h2, h1 = h1, h
        out[part] = best.cpu().numpy()
    return out


def exact(case, seed):
    if case["op"] not in ("search", "noalloc", "device") or _cells(case) > 6e9:
        return None
    if case["long_records"] or case["records"] > 25_000:
        return None
    queries, res, off, _ = _inputs(case, seed)
    all_scores = []
    for q in queries:
        sc = _exact_scores(q, res, off, _matrix(case), case["gap_open"], case["gap_extend"])
        all_scores.append(np.minimum(sc, 65535) if case["cap"] else sc)
    if case["op"] != "search":
        return {"scores": np.stack(all_scores) if case["op"] == "device" else all_scores[0]}
    sc = all_scores[0]
    best = np.lexsort((np.arange(len(sc)), -sc))[:case["top_k"]]
    out = {"hits": _hit_table([[(int(sc[i]), int(i)) for i in best if sc[i] > 0]], case["top_k"])}
    if case["scores"]:
        out["scores"] = sc
    return out
