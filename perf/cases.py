"""Workloads that the performance of the framework is judged by.

Each case is one thing that a program using the framework does through its
public entry points, at the sizes of the benchmark configurations (protein
queries of median 250 residues, PSSM queries of 50 to 2,000 rows, 300
candidates a query, exhaustive 200 x 20,000 scoring, long targets with bands,
10^6 to 10^7 seed hits, whole searches, per-profile calibration) and at the
small ends of the same ranges.  `listed()` names the cases, `draw(rng)` gives
others of the same ranges, `prepare` makes a program's state, `run` is one pass,
`work` what one pass cannot do without and `exact` the same results from plain
torch in 64 bits.
"""
import math

import numpy as np
import torch

from sabertooth_b200 import Context, GapCosts, PrefilterParams
from sabertooth_b200.api import QueryProfile
from sabertooth_b200.dtypes import HIT_DTYPE, PAIR_DTYPE, SEED_HIT_DTYPE
from sabertooth_b200.matrix import blosum62

GAPS = {"seq": (11, 1), "pssm": (44, 4)}  # the framework's default gap costs of sequence and PSSM queries


# ---- the cases ---------------------------------------------------------------
def listed():
    return [
        # the drop-in call of an unmodified caller: one query, one candidate, one answer (latency)
        {"name": "call_250x300", "kind": "call", "rows": "seq", "m": 250, "n": 300},
        # an interactive search's scoring: one query against its 300 candidates
        {"name": "one_query_300", "kind": "pairs", "rows": "seq", "queries": 1, "per_query": 300, "targets": 4000},
        # a batch of new PSSM queries: profiles made, their candidates scored, profiles freed
        {"name": "new_queries_100", "kind": "batch", "rows": "pssm", "queries": 100, "per_query": 300,
         "targets": 15000},
        # the headline batch: 4,000 PSSM queries x 300 candidates, a captured plan over device buffers
        {"name": "plan_pssm_4000", "kind": "plan", "rows": "pssm", "queries": 4000, "per_query": 300,
         "targets": 15000},
        # every query against every target, host pairs in and scores out
        {"name": "exhaustive_200", "kind": "pairs", "rows": "seq", "queries": 200, "per_query": 20000,
         "targets": 20000},
        # long targets: most pairs in a band of radius 64 around their diagonal, the others whole
        {"name": "long_mix_5000", "kind": "mix", "rows": "seq", "pairs": 5000, "radius": 64},
        # the reported hits of a search: score, start and end of every alignment
        {"name": "spans_4000", "kind": "span", "rows": "seq", "queries": 40, "per_query": 100, "targets": 4000},
        # diagonal scoring of the prefilter's seed hits, device buffers
        {"name": "hits_8M", "kind": "hits", "hits": 8000000, "queries": 400, "targets": 150000},
        # seed hits to ranked candidates (evidence, chains, gate), device buffers
        {"name": "gate_8M", "kind": "gate", "hits": 8000000, "queries": 400, "targets": 150000, "regions": True},
        # the prefilter of one query (latency) and of a batch of queries, from residues to candidates
        {"name": "search_1", "kind": "search", "rows": "seq", "queries": 1, "targets": 100000},
        {"name": "search_150", "kind": "search", "rows": "seq", "queries": 150, "targets": 300000},
        # the statistics of a PSSM search: every profile against the background samples, Gumbel fits
        {"name": "calibrate_64", "kind": "calibrate", "profiles": 64, "samples": 1000},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["call", "pairs", "batch", "plan", "mix", "span", "hits", "gate", "search", "calibrate"])
    rows = rng.choice(["seq", "pssm"])
    if kind == "call":
        return {"kind": kind, "rows": rows, "m": _log(rng, 30, 2000), "n": _log(rng, 30, 5000)}
    if kind in ("pairs", "batch", "plan"):
        q = _log(rng, 1, 600)
        return {"kind": kind, "rows": rows, "queries": q, "per_query": _log(rng, 20, min(2000, 600000 // q)),
                "targets": _log(rng, 2000, 20000)}
    if kind == "mix":
        return {"kind": kind, "rows": rows, "pairs": _log(rng, 50, 5000), "radius": _log(rng, 16, 128)}
    if kind == "span":
        q = _log(rng, 1, 100)
        return {"kind": kind, "rows": rows, "queries": q, "per_query": _log(rng, 5, 4000 // q), "targets": 4001}
    if kind == "hits":
        return {"kind": kind, "hits": _log(rng, 20000, 8000000), "queries": _log(rng, 10, 1000), "targets": 60001}
    if kind == "gate":
        return {"kind": kind, "hits": _log(rng, 20000, 8000000), "queries": _log(rng, 10, 1000), "targets": 60001,
                "regions": rng.random() < 0.5}
    if kind == "search":
        return {"kind": kind, "rows": "seq", "queries": _log(rng, 1, 150), "targets": _log(rng, 20000, 300000)}
    p = _log(rng, 2, 64)
    return {"kind": kind, "profiles": p, "samples": _log(rng, 50, 1000)}


# ---- inputs --------------------------------------------------------------------
_MAT = blosum62()
_BACK = np.asarray(_MAT.p_back[:20], dtype=np.float64)
_BACK = _BACK / _BACK.sum()
_LUT = np.searchsorted(np.cumsum(_BACK), (np.arange(65536) + 0.5) / 65536.0).clip(0, 19).astype(np.uint8)


def _background(rng, n):
    """n residues of the background composition."""
    return _LUT[rng.integers(0, 65536, n, dtype=np.uint16)]


def _lognormal(rng, n, median, sigma, lo, hi):
    return np.clip(np.rint(median * np.exp(sigma * rng.standard_normal(n))), lo, hi).astype(np.int64)


def _query_lengths(rng, n, rows):
    if rows == "seq":
        return _lognormal(rng, n, 250, 0.5, 30, 1000)
    return np.rint(np.exp(rng.uniform(math.log(50), math.log(2000), n))).astype(np.int64)


def _offsets(lens):
    o = np.zeros(len(lens) + 1, dtype=np.int64)
    o[1:] = np.cumsum(lens)
    return o


def _rows(rng, residues, rows):
    """int32 [n][21] score rows: BLOSUM62, or position-specific rows of the same consensus with the spread of
    family PSSMs (three times the matrix, about -11 on average, clipped to the range that they have)."""
    r = np.asarray(_MAT.sequence_rows(residues), dtype=np.int32).reshape(-1, 21)
    if rows == "pssm":
        r = np.clip(3 * r - 7 + np.rint(4.0 * rng.standard_normal(r.shape)).astype(np.int32), -30, 48)
        r[:, 20] = 0
    return np.ascontiguousarray(r, dtype=np.int32)


def _plant(rng, arena, toff, ti, qres, qoff, qi, keep):
    """Copies a random stretch of query qi[k] over a random stretch of target ti[k], each site kept with
    probability `keep`; returns (target start - query start, query start, length) of each."""
    ql, tl = np.diff(qoff)[qi], np.diff(toff)[ti]
    ln = np.minimum(ql, tl)
    qs = (rng.random(len(ti)) * (ql - ln + 1)).astype(np.int64)
    ts = (rng.random(len(ti)) * (tl - ln + 1)).astype(np.int64)
    o = _offsets(ln)
    j = np.arange(o[-1]) - np.repeat(o[:-1], ln)
    src = qres[np.repeat(qoff[:-1][qi] + qs, ln) + j]
    dst = np.repeat(toff[:-1][ti] + ts, ln) + j
    k = rng.random(len(dst)) < keep
    arena[dst[k]] = src[k]
    return ts - qs, qs, ln


def _inputs(case, seed):
    """The host side of a case: query residues and rows, database, and what the kind adds."""
    rng = np.random.default_rng([int(seed), 77])
    kind, rows = case["kind"], case.get("rows", "seq")
    w = {"kind": kind, "gaps": GAPS["pssm" if kind == "calibrate" else rows]}
    if kind == "call":
        ql, tl = np.array([case["m"]]), np.array([case["n"]])
    elif kind == "calibrate":
        rows = "pssm"
        ql, tl = _query_lengths(rng, case["profiles"], rows), _lognormal(rng, 2000, 250, 0.4, 30, 1000)
    elif kind == "mix":
        n = case["pairs"]
        ql = _lognormal(rng, n, 250, 0.5, 30, 2000)
        longer = rng.random(n) < 0.1
        tl = np.exp(np.where(longer, rng.uniform(math.log(10001), math.log(35000), n),
                             rng.uniform(math.log(1000), math.log(10000), n))).astype(np.int64)
    elif kind in ("hits", "gate"):
        ql, tl = _query_lengths(rng, case["queries"], "seq"), _lognormal(rng, case["targets"], 160, 0.55, 30, 1000)
    else:
        ql = _query_lengths(rng, case["queries"], rows)
        med, sig = (160, 0.55) if rows == "pssm" else (250, 0.35 if kind == "search" else 0.5)
        tl = _lognormal(rng, case["targets"], med, sig, 30, 1000)
    qoff, toff = _offsets(ql), _offsets(tl)
    qres, arena = _background(rng, int(qoff[-1])), _background(rng, int(toff[-1]))
    w.update(qres=qres, qoff=qoff, arena=arena, toff=toff, rows=_rows(rng, qres, rows))
    nq, nt = len(ql), len(tl)
    # homologs: a tenth of the targets (the mix: each twentieth pair nearly identical; a search: five per query)
    if kind == "mix":
        ti = np.nonzero(rng.random(nt) < 0.05)[0]
        qi, keep = ti, 0.97
    elif kind == "call":
        ti, qi, keep = np.zeros(1, np.int64), np.zeros(1, np.int64), 0.4
    elif kind == "search":
        ti = rng.permutation(nt)[:5 * nq]
        qi, keep = np.arange(len(ti)) % nq, 0.5
    elif kind == "calibrate":
        ti, qi, keep = np.zeros(0, np.int64), np.zeros(0, np.int64), 0.0
    else:
        ti = np.nonzero(rng.random(nt) < 0.1)[0]
        qi, keep = rng.integers(0, nq, len(ti)), 0.45
    diag, qs, ln = _plant(rng, arena, toff, ti, qres, qoff, qi, keep)
    if kind in ("pairs", "batch", "plan", "span"):
        per = min(case["per_query"], nt)
        if per == nt:
            pt = np.tile(np.arange(nt, dtype=np.uint32), nq)
        else:
            pt = np.concatenate([rng.permutation(nt)[:per] for _ in range(nq)]).astype(np.uint32)
            k = rng.random(len(ti)) < 0.5  # half of the homologs are among their query's candidates
            pt[qi[k] * per + rng.integers(0, per, int(k.sum()))] = ti[k]
        w.update(pq=np.repeat(np.arange(nq, dtype=np.uint32), per), pt=pt)
    elif kind == "mix":
        center = np.zeros(nt, np.int32)
        center[ti] = diag
        w.update(pq=np.arange(nq, dtype=np.uint32), pt=np.arange(nt, dtype=np.uint32), center=center,
                 radius=np.where(tl > 4 * ql, case["radius"], -1).astype(np.int32))
    elif kind in ("hits", "gate"):
        n = case["hits"]
        nh = 3 * n // 10 if len(ti) else 0  # three tenths on or beside the homologs' diagonals
        h = rng.integers(0, max(len(ti), 1), nh)
        jitter = rng.integers(-3, 4, nh) if kind == "hits" else 6 * (rng.random(nh) < 0.3)
        rq, rt = rng.integers(0, nq, n - nh), rng.integers(0, nt, n - nh)
        rd = (rng.random(n - nh) * (ql[rq] + tl[rt] - 1)).astype(np.int64) - ql[rq] + 1
        q, t, d = np.concatenate([qi[h], rq]), np.concatenate([ti[h], rt]), np.concatenate([diag[h] + jitter, rd])
        if kind == "hits":  # in the prefilter's order
            s = torch.from_numpy(((q * nt + t) << 12) + d + 1024)
            o = torch.argsort(s.cuda()).cpu().numpy() if torch.cuda.is_available() else torch.argsort(s).numpy()
            w.update(hq=q[o], ht=t[o], hd=d[o])
        else:  # a position of the diagonal's overlap that the planted stretch or the whole diagonal holds
            lo, hi = np.maximum(-d, 0), np.minimum(ql[q], tl[t] - d)
            lo[:nh], hi[:nh] = np.maximum(lo[:nh], qs[h]), np.minimum(hi[:nh], qs[h] + ln[h])
            hi = np.maximum(hi, lo + 1)
            o = rng.permutation(n)
            qp = lo + (rng.random(n) * (hi - lo)).astype(np.int64)
            ok = (qp < ql[q]) & (qp + d >= 0) & (qp + d < tl[t])
            qp = np.where(ok, qp, np.maximum(-d, 0))
            ok = (qp < ql[q]) & (qp + d >= 0) & (qp + d < tl[t])
            d, qp = np.where(ok, d, 0), np.where(ok, qp, 0)
            w.update(hq=q[o], ht=t[o], hd=d[o], hp=qp[o])
    return w


# ---- a program's state and one pass -----------------------------------------------
_stream = None


def _device_stream():
    """One stream for the calls that return before the GPU is done, as a program has one."""
    global _stream
    if _stream is None:
        _stream = torch.cuda.Stream()
    return _stream


def _pairs(w, ids):
    p = np.zeros(len(w["pq"]), dtype=PAIR_DTYPE)
    p["profile"] = ids[w["pq"]]
    p["target"] = w["pt"]
    p["band_center"] = w.get("center", 0)
    p["band_radius"] = w.get("radius", -1)
    return p


def prepare(case, seed):
    w = _inputs(case, seed)
    kind = case["kind"]
    gaps = GapCosts(*w["gaps"])
    ctx = Context(0)
    s = {"kind": kind, "ctx": ctx, "gaps": gaps}
    if kind == "call":
        s.update(query=QueryProfile.from_rows(w["rows"], ctx), target=w["arena"])
        return s
    ctx.upload_db(w["arena"], w["toff"].astype(np.uint64))
    if kind in ("plan", "hits", "gate"):
        ctx.set_stream(_device_stream().cuda_stream)
    if kind == "batch":  # the rows stay on the host: making their profiles is part of a pass
        s.update(rows=w["rows"], offsets=w["qoff"].astype(np.uint64), w=w, pairs=_pairs(w, np.arange(case["queries"])))
        return s
    ids = ctx.create_profiles_arena(w["rows"], w["qoff"].astype(np.uint64))
    if kind in ("pairs", "mix", "span"):
        s["pairs"] = _pairs(w, ids)
    elif kind == "plan":
        pairs = _pairs(w, ids)
        s["scores"] = torch.zeros(len(pairs), dtype=torch.int32, device="cuda")
        s["plan"] = ctx.plan(pairs, gaps, s["scores"].data_ptr())
    elif kind in ("hits", "gate"):
        n = len(w["hq"])
        h = np.zeros(n, dtype=HIT_DTYPE if kind == "hits" else SEED_HIT_DTYPE)
        h["query"], h["target"], h["diag"] = ids[w["hq"]], w["ht"], w["hd"]
        if kind == "gate":
            h["qpos"] = w["hp"]
            s["params"] = PrefilterParams(regions=bool(case["regions"]))
            s["out"] = torch.zeros(n * 8, dtype=torch.int32, device="cuda")  # room for n candidates, the API's bound
        else:
            s["out"] = [torch.zeros(n, dtype=torch.int32, device="cuda") for _ in range(4)]
            s["count"] = torch.zeros(1, dtype=torch.int64, device="cuda")
        s["n"] = n
        s["hits"] = torch.from_numpy(h.view(np.uint8)).cuda()
    elif kind == "search":
        ctx.seed_index_build("111001101")
        s.update(ids=ids, queries=[w["qres"][a:b] for a, b in zip(w["qoff"][:-1], w["qoff"][1:])],
                 params=PrefilterParams(min_diag_score=43, span=9),
                 found=np.zeros((1024 * case["queries"], 8), dtype=np.int32))  # room for a batch's candidates
    else:
        s.update(ids=ids, lengths=np.diff(w["toff"]).astype(np.uint32), samples=case["samples"])
    torch.cuda.synchronize()
    return s


def run(s):
    kind, ctx, gaps = s["kind"], s["ctx"], s["gaps"]
    if kind == "call":
        score, kernel = s["query"].sw_score_with(s["target"], gaps)
        return {"score": score, "kernel": int(kernel)}
    if kind == "batch":
        ids = ctx.create_profiles_arena(s["rows"], s["offsets"])
        pairs = s["pairs"].copy()
        pairs["profile"] = ids[pairs["profile"]]
        scores, kernels = ctx.sw_score_pairs(pairs, gaps, with_kernels=True)
        ctx.free_profiles(ids)
        return {"scores": scores, "kernels": kernels}
    if kind in ("pairs", "mix"):
        return {"scores": ctx.sw_score_pairs(s["pairs"], gaps)}
    if kind == "plan":
        s["plan"].run()
        return {"scores": s["scores"]}
    if kind == "span":
        scores, starts, ends = ctx.align_span_pairs(s["pairs"], gaps)
        return {"scores": scores, "starts": starts, "ends": ends}
    if kind == "hits":
        a, b, q, t = s["out"]
        ctx.ungapped_hits_device(s["hits"].data_ptr(), s["n"], a.data_ptr(), b.data_ptr(), q.data_ptr(), t.data_ptr(),
                                 s["count"].data_ptr())
        return {"per_hit": a, "pair_best": b, "pair_query": q, "pair_target": t, "pairs": s["count"]}
    if kind == "gate":
        n, counters = ctx.prefilter_gate_device(s["hits"].data_ptr(), s["n"], s["out"].data_ptr(), s["params"], gaps)
        return {"candidates": s["out"], "kept": n, "counters": counters}
    if kind == "search":
        found, evidence, seeds = ctx.prefilter_queries(s["ids"], s["queries"], s["params"], gaps)
        s["found"][:len(found)] = found.view(np.int32).reshape(-1, 8)
        return {"candidates": s["found"], "kept": len(found), "evidence": evidence, "seeds": seeds}
    fits, scores = ctx.calibrate_profiles(s["ids"], s["lengths"], s["samples"], gaps=gaps, with_scores=True)
    return {"fits": np.array([f or (math.nan,) * 3 for f in fits]), "scores": scores}


# ---- what a pass cannot do without ---------------------------------------------------
def work(case):
    """Inputs read once and outputs written once; a dynamic-programming cell is two additions and four maxima
    of Gotoh's recurrence, a diagonal's cell one addition and two maxima.  Sizes are the expected ones."""
    kind, rows = case["kind"], case.get("rows", "seq")
    m = {"seq": 280.0, "pssm": 528.0}[rows]
    t = 185.0 if rows == "pssm" or kind in ("hits", "gate") else 265.0 if kind == "search" else 280.0
    if kind == "call":
        return {"bytes": 22.0 * case["m"] + case["n"] + 8, "flops": 6.0 * case["m"] * case["n"]}
    if kind in ("pairs", "batch", "plan", "span"):
        n = float(case["queries"] * min(case["per_query"], case["targets"]))
        row_bytes = 84.0 if kind == "batch" else 21.0  # new queries come as 32-bit rows
        out = 20.0 if kind == "span" else 8.0 if kind == "batch" else 4.0
        return {"bytes": case["queries"] * m * row_bytes + min(case["targets"], n) * t + n * (16 + out),
                "flops": 6.0 * n * m * t * (1.4 if kind == "span" else 1.0)}  # the start pass: the prefix's cells
    if kind == "mix":
        n = float(case["pairs"])
        # nine tenths of the pairs hold 2 radius + 1 cells a row; a whole pair about 600 x 1,500
        return {"bytes": n * (280 * 21.0 + 6300 + 20),
                "flops": 6.0 * n * (0.92 * 280 * (2 * case["radius"] + 1) + 0.08 * 600 * 1500)}
    if kind == "hits":
        return {"bytes": case["hits"] * (12.0 + 4.0 + 12.0) + case["targets"] * t, "flops": 3.0 * 115 * case["hits"]}
    if kind == "gate":
        return {"bytes": case["hits"] * 16.0 + case["targets"] * t, "flops": 3.0 * 75 * case["hits"]}
    if kind == "search":
        # about 1,150 postings of 8 bytes a query and million residues, a window of 105 cells for each
        hits = case["queries"] * 1150.0 * case["targets"] * t / 1e6
        return {"bytes": hits * 8.0 + case["targets"] * t + case["queries"] * m * 22, "flops": 3.0 * 105 * hits}
    n = float(case["profiles"] * case["samples"])
    return {"bytes": case["profiles"] * 528 * 21.0 + case["samples"] * 270.0 + 4 * n, "flops": 6.0 * n * 528 * 270}


# ---- the same results in plain torch, 64 bits ------------------------------------------
def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _gotoh(prof, q, codes, n, m, gaps, band=None, rev=None):
    """Smith-Waterman-Gotoh over a batch of pairs: (best, end row, end column), the first optimum by column,
    then row.  prof [nq, 22, M]; codes [B, N] (21 past the end); band (center, radius); rev: each pair's last
    query row, whose rows run backwards from there."""
    go, ge = gaps
    dev, B, M = prof.device, len(q), prof.shape[2]
    i = torch.arange(M, device=dev)
    H = torch.zeros(B, M, dtype=torch.int64, device=dev)
    E = torch.full_like(H, -go)
    best, br, bc = (torch.zeros(B, dtype=torch.int64, device=dev) for _ in range(3))
    if rev is not None:
        at = (rev[:, None] - i).clamp(min=0)
        live = i <= rev[:, None]
    for j in range(int(n.max()) if B else 0):
        S = prof[q, codes[:, j].long()].long()
        if rev is not None:
            S = torch.where(live, S.gather(1, at), torch.zeros_like(S))
        d = torch.zeros_like(H)
        d[:, 1:] = H[:, :-1]
        x = torch.maximum(d + S, E).clamp(min=0)
        if band is not None:
            inside = (j - i - band[0][:, None]).abs() <= band[1][:, None]
            x = torch.where(inside, x, torch.zeros_like(x))
        F = torch.full_like(H, -go)
        F[:, 1:] = torch.cummax(x + i * ge, 1).values[:, :-1] - go - i[:-1] * ge
        H = torch.maximum(x, F)
        E = torch.maximum(E - ge, H - go)
        if band is not None:
            H = torch.where(inside, H, torch.zeros_like(H))
            E = torch.where(inside, E, torch.full_like(E, -go))
        top = H.amax(1)
        up = (top > best) & (j < n)
        row = torch.where(H == top[:, None], i, M).amin(1)
        best, br, bc = torch.where(up, top, best), torch.where(up, row, br), torch.where(up, torch.full_like(bc, j), bc)
    return best, br, bc


def _profiles(w, dev):
    ql = np.diff(w["qoff"])
    p = torch.zeros(len(ql), int(ql.max()), 22, dtype=torch.int32)
    for k, (a, b) in enumerate(zip(w["qoff"][:-1], w["qoff"][1:])):
        p[k, :b - a, :21] = torch.from_numpy(w["rows"][a:b])
    return p.permute(0, 2, 1).contiguous().to(dev)


def _codes(arena, off, tl, N, dev):
    j = torch.arange(N, device=dev)
    at = (off[:, None] + j).clamp(max=len(arena) - 1)
    return torch.where(j < tl[:, None], arena[at], torch.full((), 21, dtype=torch.uint8, device=dev))


def _score_pairs(w, pq, pt, arena, toff, spans=False):
    """Scores (and spans) of all pairs, in chunks of similar size; None where that would take too long."""
    dev = _dev()
    ql, tl = np.diff(w["qoff"])[pq], np.diff(toff)[pt]
    o = np.lexsort((tl, ql)) if "center" not in w else np.lexsort((ql, tl))
    chunks, a = [], 0
    while a < len(o):
        b = min(len(o), a + max(64, int(3e7 // max(int(ql[o[a:a + 4096]].max()), 1))))
        chunks.append(o[a:b])
        a = b
    cost = sum(float(tl[c].max()) * (150e-6 + 25.0 * len(c) * float(ql[c].max()) * 8 / 3e12) for c in chunks)
    if cost * (2 if spans else 1) > 15 or dev.type == "cpu" and cost > 0.2:
        return None
    prof, mem = _profiles(w, dev), torch.from_numpy(arena).to(dev)
    out = np.zeros((len(pq), 5), dtype=np.int64)
    for c in chunks:
        M, N = int(ql[c].max()), int(tl[c].max())
        q = torch.from_numpy(pq[c].astype(np.int64)).to(dev)
        n, m = torch.from_numpy(tl[c]).to(dev), torch.from_numpy(ql[c]).to(dev)
        codes = _codes(mem, torch.from_numpy(toff[:-1][pt[c]]).to(dev), n, N, dev)
        band = None
        if "center" in w:
            wide = torch.full((len(c),), 1 << 40, device=dev)
            r = torch.from_numpy(w["radius"][c].astype(np.int64)).to(dev)
            band = (torch.from_numpy(w["center"][c].astype(np.int64)).to(dev), torch.where(r < 0, wide, r))
        s, er, ec = _gotoh(prof[:, :, :M], q, codes, n, m, w["gaps"], band)
        got = [s, torch.where(s > 0, er, -1), torch.where(s > 0, ec, -1)]
        if spans:
            k = torch.arange(N, device=dev)
            back = codes.gather(1, (ec[:, None] - k).clamp(min=0))
            back = torch.where(k <= ec[:, None], back, torch.full_like(back, 21))
            _, fr, fc = _gotoh(prof[:, :, :M], q, back, ec + 1, m, w["gaps"], rev=er)
            got += [torch.where(s > 0, er - fr, -1), torch.where(s > 0, ec - fc, -1)]
        out[c, :len(got)] = torch.stack(got, 1).cpu().numpy()
    return out


def _mix64(z):
    z = (z ^ (z >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
    z = (z ^ (z >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
    return z ^ (z >> np.uint64(31))


def _samples(lengths, count, seed=0x5EED):
    """The background targets: sample i draws its length, then its residues, from its own SplitMix64 stream."""
    g = np.uint64(0x9E3779B97F4A7C15)
    cum = np.cumsum(np.asarray(_MAT.p_back[:20], dtype=np.float64) / math.fsum(_MAT.p_back[:20]))
    cum[-1] = 1.0
    seqs = []
    with np.errstate(over="ignore"):
        for i in range(count):
            s = np.uint64(seed) ^ (np.uint64(0xBEEF) * np.uint64(0xA24BAED4963EE407))
            s = _mix64((s ^ (np.uint64(i) * np.uint64(0x9FB21C651E98DF25))) + g) + g
            n = max(int(lengths[int(_mix64(s) % np.uint64(len(lengths)))]), 1)
            u = _mix64(s + np.arange(1, n + 1, dtype=np.uint64) * g) >> np.uint64(11)
            seqs.append(np.searchsorted(cum, u.astype(np.float64) / float(1 << 53), side="right").astype(np.uint8))
    return seqs


def _gumbel(x):
    """Maximum-likelihood Gumbel parameters (lambda, mu): the root of the profile likelihood's derivative."""
    mean, lo = x.mean(), x.min()
    lam = math.pi / math.sqrt(6.0 * x.var(ddof=1))
    for _ in range(100):
        e = np.exp(-lam * (x - lo))
        s0, s1, s2 = e.sum(), (x * e).sum(), (x * x * e).sum()
        f, df = 1.0 / lam - mean + s1 / s0, -1.0 / lam**2 - s2 / s0 + (s1 / s0) ** 2
        step = f / df
        lam = lam - step if lam > step else lam / 2
        if abs(step) < 1e-15 * lam:
            break
    return lam, lo - math.log(np.exp(-lam * (x - lo)).mean()) / lam


def _kadane(w):
    dev = _dev()
    n = len(w["hq"])
    if dev.type == "cpu" and n > 50000:
        return None
    prof, mem = _profiles(w, dev), torch.from_numpy(w["arena"]).to(dev)
    qoff, toff = (torch.from_numpy(w[k]).to(dev) for k in ("qoff", "toff"))
    out = []
    for a in range(0, n, 1 << 20):
        q, t, d = (torch.from_numpy(w[k][a:a + (1 << 20)].astype(np.int64)).to(dev) for k in ("hq", "ht", "hd"))
        lo = (-d).clamp(min=0)
        hi = torch.minimum(qoff[q + 1] - qoff[q], toff[t + 1] - toff[t] - d)
        cur = torch.zeros_like(q)
        best = torch.zeros_like(q)
        for k in range(int((hi - lo).clamp(min=0).max())):
            i = lo + k
            live = i < hi
            j = torch.where(live, i, lo).clamp(max=prof.shape[2] - 1)
            r = mem[(toff[t] + j + d).clamp(0, len(mem) - 1)].long()
            cur = cur.clamp(min=0) + torch.where(live, prof[q, r, j].long(), torch.zeros_like(q))
            best = torch.maximum(best, cur)
        out.append(best.cpu().numpy())
    return np.concatenate(out)


def exact(case, seed):
    """Scores, ends, starts, diagonal scores and Gumbel fits.  Kernel tags, run lists, candidates and counters
    have no value of their own here (they are whole numbers)."""
    kind = case["kind"]
    if kind in ("gate", "search"):
        return None
    w = _inputs(case, seed)
    if kind == "hits":
        return {"per_hit": _kadane(w), "pair_best": None, "pair_query": None, "pair_target": None, "pairs": None}
    if kind == "call":
        out = _score_pairs(w, np.zeros(1, np.int64), np.zeros(1, np.int64), w["arena"], w["toff"])
        return None if out is None else {"score": int(out[0, 0]), "kernel": None}
    if kind == "calibrate":
        lengths = np.diff(w["toff"])
        seqs = _samples(lengths, case["samples"])
        ql, count = np.diff(w["qoff"]), case["samples"]
        pq, pt = np.repeat(np.arange(len(ql)), count), np.tile(np.arange(count), len(ql))
        out = _score_pairs(w, pq, pt, np.concatenate(seqs), _offsets([len(s) for s in seqs]))
        if out is None:
            return None
        sc = out[:, 0].reshape(len(ql), count)
        fits = []
        for x, m in zip(sc.astype(np.float64), ql):
            lam, mu = _gumbel(x)
            fits.append((lam, math.exp(lam * (mu + 0.5)) / (float(m) * lengths.mean()), mu))
        return {"fits": np.array(fits), "scores": sc}
    out = _score_pairs(w, w["pq"], w["pt"], w["arena"], w["toff"], spans=kind == "span")
    if out is None:
        return None
    if kind == "span":
        return {"scores": out[:, 0], "starts": out[:, 3:5], "ends": out[:, 1:3]}
    return {"scores": out[:, 0], "kernels": None} if kind == "batch" else {"scores": out[:, 0]}
