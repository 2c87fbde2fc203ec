"""Timed cases of the word-hit stage: what a program that uses the library has
it do, from host queries to ordered HSPs on the host.

A case names a way of calling the library (`call`), the queries and the
database.  Databases have the length law of the benchmark's synthetic
workloads (lognormal, median 300, sigma 0.6, 30..5000) with 1 % of the
subjects carrying a mutated segment of a query, so that extensions, kept HSPs
and the ordering pass are exercised as in a real search.

    search    queries arrive on the host: build their lookup tables, search,
              bring the ordered HSPs and counters back (the usual call)
    resident  the batch is kept, only the search is repeated (`Searcher`)
    served    requests submitted one by one to the continuous-batching server
    open      a database is opened from host arrays and searched once

Results are whole numbers, equal on every correct implementation, so there is
no 64-bit restatement of them here.
"""
import ctypes as C
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "h-blast_gb300"))
import hblast  # noqa: E402
from hblast import synth  # noqa: E402

HSP_BYTES = 36
MEAN_SUBJECT = 360          # mean letters of a subject under the length law above
# the most work of a drawn case: query letters x subject letters of batch64_500k
MOST_CELLS = 64 * 775 * 500_000 * MEAN_SUBJECT


def case(name, call, program, law, lo, hi, queries, subjects, threshold=11, window=40, group_len=0, seg=False):
    d = {"call": call, "program": program, "law": law, "lo": lo, "hi": hi, "queries": queries, "subjects": subjects,
         "threshold": threshold, "window": window, "group_len": group_len, "seg": seg}
    return {"name": name, **d} if name else d


def listed():
    return [
        # a script that compares one protein with a handful of others: latency only
        case("one_300_vs_400", "search", "blastp", "uniform", 300, 300, 1, 400),
        # the shortest query the workloads have, against a small proteome
        case("peptide_30_vs_20k", "search", "blastp", "uniform", 30, 30, 1, 20_000),
        # the plain configuration: one protein against one proteome
        case("plain_300_vs_20k", "search", "blastp", "uniform", 300, 300, 1, 20_000),
        # interactive search of one protein against a reviewed-proteins-sized database
        case("one_350_vs_300k", "search", "blastp", "uniform", 350, 350, 1, 300_000),
        # a file of proteins with heavy-tailed lengths
        case("tail8_vs_200k", "search", "blastp", "heavy", 30, 35_000, 8, 200_001),
        # the batched configuration's queries on a quarter of its database: the largest
        case("batch64_vs_500k", "search", "blastp", "uniform", 50, 1500, 64, 500_000),
        # nucleotide reads and transcripts, six frames, SEG-masked as blastx does
        case("blastx8_seg_vs_100k", "search", "blastx", "uniform", 300, 3000, 8, 100_003, seg=True),
        # one giant protein (titin-like)
        case("long_20000_vs_20k", "search", "blastp", "uniform", 20_000, 20_000, 1, 20_000),
        # a kept batch searched again and again: device time without the table build
        case("resident16_vs_200k", "resident", "blastp", "uniform", 50, 1500, 16, 200_000),
        # other word threshold, two-hit window and group length, all offered as options
        case("options_t12_w60_vs_100k", "search", "blastp", "uniform", 100, 900, 12, 99_991, threshold=12, window=60,
             group_len=2008),
        # a service: mixed requests batched as they arrive
        case("served24_vs_100k", "served", "mixed", "heavy", 30, 4000, 24, 100_000),
        # the command-line program: open the database, search one protein
        case("open_50k_search", "open", "blastp", "uniform", 433, 433, 1, 50_000),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    call = rng.choice(["search"] * 7 + ["resident"] * 3 + ["served"] + ["open"])
    program = "mixed" if call == "served" else rng.choice(["blastp", "blastp", "blastp", "blastx"])
    law = rng.choice(["uniform", "heavy"]) if program == "blastp" else ("uniform" if program == "blastx" else "heavy")
    if program == "blastx":
        lo, hi, queries = 300, 3000, _log_int(rng, 1, 32)
        mean = 2 * 1650
    elif program == "mixed":
        lo, hi, queries = 30, 4000, _log_int(rng, 4, 48)
        mean = 900
    elif law == "heavy":
        lo, hi, queries = 30, 35_000, _log_int(rng, 1, 32)
        mean = 700
    else:
        lo = _log_int(rng, 30, 1500)
        hi = min(35_000, max(lo, int(lo * rng.uniform(1.0, 4.0))))
        queries = _log_int(rng, 1, 64)
        mean = (lo + hi) // 2
    most = 100_000 if call in ("open", "served") else 500_000
    most = max(200, min(most, MOST_CELLS // 2 // (mean * queries * MEAN_SUBJECT)))
    subjects = _log_int(rng, 100, most) if most > 100 else 100
    threshold = rng.choice([11, 11, 11, 12, 13])
    window = rng.choice([40, 40, 40, 20, 60])
    group_len = rng.choice([0, 0, 0, 1000, 2008])
    if call == "served":
        threshold, window, group_len = 11, 40, 0
    return case(None, call, program, law, lo, hi, queries, subjects, threshold, window, group_len,
                seg=program == "blastx" and rng.random() < 0.5)


def _lengths(c):
    """Query lengths of a case: evenly spread quantiles of its law, so that they
    depend on the case alone and the letters on the seed."""
    n = c["queries"]
    u = (np.arange(n) + 0.5) / n
    if c["law"] == "heavy":
        z = np.sqrt(2.0) * torch.erfinv(torch.from_numpy(2 * u - 1)).numpy()
        lens = np.clip(np.rint(350 * np.exp(z)), c["lo"], c["hi"])
    else:
        lens = np.rint(c["lo"] + u * (c["hi"] - c["lo"]))
    return np.random.default_rng(n).permutation(lens.astype(np.int64))


def _query_letters(c):
    lens = _lengths(c)
    if c["program"] == "blastx":
        return int(2 * lens.sum())
    return int(lens.sum()) + (900 * c["queries"] if c["program"] == "mixed" else 0)


def _expected_hsps(c):
    return 1.6e-7 * _query_letters(c) * c["subjects"] * MEAN_SUBJECT + 0.01 * c["subjects"]


def _nucleotides(rng, db, lens):
    """Random nucleotide queries, each with a mutated, back-translated piece of a subject in it."""
    out = []
    for n in lens:
        nt = rng.integers(0, 4, size=int(n), dtype=np.uint8)
        s = db.subject(int(rng.integers(db.n)))
        orf = min(len(s), int(n) // 4, 300)
        cod = synth.back_translate(rng, synth.mutate(rng, s[:orf], rng.uniform(0.40, 0.70)))
        if rng.random() < 0.5:
            cod = (3 - cod[::-1]).astype(np.uint8)
        at = int(rng.integers(0, len(nt) - len(cod) + 1))
        nt[at:at + len(cod)] = cod
        out.append(nt)
    return out


def prepare(c, seed):
    rng = np.random.default_rng([seed, c["queries"], c["subjects"]])
    donors = [synth.random_letters(rng, int(n)) for n in _lengths(c)]
    db = synth.make_db(rng, c["subjects"], 300, 0.6, 30, 5000, 0.01, donors,
                       lambda r: r.integers(50, 301), lambda r: r.uniform(0.30, 0.60))
    if c["program"] == "blastx":
        queries = _nucleotides(rng, db, _lengths(c))
    else:
        queries = [hblast.ProteinQuery.blastp(d) for d in donors]
    if c["program"] == "mixed":           # four proteins to one nucleotide query
        for i in range(4, len(queries), 5):
            queries[i] = _nucleotides(rng, db, [1650])[0]
    # the caller's buffers: ordered HSPs and per-query counters
    state = {"case": c, "queries": queries,
             "hsps": np.zeros((int(2 * _expected_hsps(c)) + 4096, HSP_BYTES // 4), np.int32),
             "stats": np.zeros((len(queries), len(_STATS)), np.int64)}
    if c["call"] == "open":
        state["residues"], state["offsets"] = db.residues, db.offsets
        return state
    state["db"] = hblast.Database(db.residues, db.offsets)
    if c["call"] == "resident":
        state["batch"] = _batch(c, queries)
        state["stream"] = torch.cuda.Stream()
        state["searcher"] = hblast.Searcher(state["db"], state["batch"])
    if c["call"] == "served":
        state["server"] = hblast.Server(state["db"])
    return state


def _batch(c, queries):
    if c["program"] == "blastx":
        n = len(queries)
        return hblast.Batch.blastx(queries, np.full((n, 6), synth.X_DROPOFF, np.int32), np.full((n, 6), synth.CUTOFF, np.int32),
                                   threshold=c["threshold"], window=c["window"], max_group_len=c["group_len"],
                                   seg=True if c["seg"] else None)
    return hblast.Batch.proteins(queries, threshold=c["threshold"], window=c["window"], max_group_len=c["group_len"])


_STATS = ("lookup_hits", "init_extends", "good_init_extends", "subjects_passed")


def _check(rc):
    if rc != 0:
        raise RuntimeError(hblast.lib().hbg_last_error().decode())


def _search(db, batch, state):
    """One search through the C ABI, straight into the caller's buffers."""
    n = C.c_int64()
    opt = hblast.default_options()
    _check(hblast.lib().hbg_search_sync(db.handle, batch.handle, C.byref(opt), state["hsps"].ctypes.data, len(state["hsps"]),
                                        C.byref(n), state["stats"].ctypes.data_as(C.POINTER(hblast.core.QueryStats)), None))
    return n.value


def run(state):
    c = state["case"]
    hsps, stats = state["hsps"], state["stats"]
    if c["call"] == "resident":
        s = state["searcher"]
        s.launch(state["stream"].cuda_stream)
        s.wait()
        n = s.n_hsps()
        _check(hblast.lib().hbg_result_hsps(s.res, 0, n, hsps.ctypes.data))
        one = hblast.core.QueryStats()
        for q in range(len(stats)):
            _check(hblast.lib().hbg_result_stats(s.res, q, C.byref(one)))
            stats[q] = [getattr(one, k) for k in _STATS]
    elif c["call"] == "served":
        srv = state["server"]
        xd, cu = np.full(6, synth.X_DROPOFF, np.int32), np.full(6, synth.CUTOFF, np.int32)
        tickets = [srv.submit(q) if isinstance(q, hblast.ProteinQuery) else srv.submit_blastx(q, xd, cu)
                   for q in state["queries"]]
        n = 0
        for q, t in enumerate(tickets):
            got, st, _ = srv.take(t)
            hsps[n:n + len(got)] = got.view(np.int32).reshape(-1, HSP_BYTES // 4)
            stats[q] = [st[k] for k in _STATS]
            n += len(got)
    else:
        db = hblast.Database(state["residues"], state["offsets"]) if c["call"] == "open" else state["db"]
        batch = _batch(c, state["queries"])
        n = _search(db, batch, state)
        batch.close()
        if c["call"] == "open":
            db.close()
    return {"n": n, "hsps": hsps, "stats": stats}


def work(c):
    """Subject letters and 8 bytes of place each, the query letters, and the HSP
    records; one word look-up per subject letter and query group of 4056 letters
    and, per lookup hit (about 1.6e-3 of the letter pairs at threshold 11), one
    update of its diagonal, as operations."""
    query = _query_letters(c)
    letters = c["subjects"] * MEAN_SUBJECT
    passes = max(1, round(query / 4056))
    per_cell = {11: 1.6e-3, 12: 1.0e-3}.get(c["threshold"], 0.6e-3)
    return {"bytes": letters + 8 * c["subjects"] + query + HSP_BYTES * _expected_hsps(c),
            "flops": passes * letters + per_cell * query * letters}
