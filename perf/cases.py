"""The measured cases: searches of genome sequence against repeat libraries through the public
Python entry points (Searcher.search / search_resident and Results.tabular).

A case names a query set, a library and the search settings:
  queries   number of query sequences (a self search takes that many of the library's consensi)
  bp        length of a query; the median where `spread` is the sigma of log-normal lengths
  spread    0: every query has `bp` bases
  library   number of library consensi (log-normal lengths, median 1.5 kb, 100-12,000 bp)
  self      the library against itself: consensi of 200-10,000 bp, a fifth of them derived from others
  word      word size
  flags     "repeatmasker": the cutoffs and X-drops RepeatMasker passes, masklevel 80 (off in a
            self search), complexity adjustment; "defaults": rmblastn's command-line defaults
  dust      DUST masking of the queries (rmblastn's own default is on; RepeatMasker's is off)
  schedule  0: records in arrival order; 1: the learned order
  pipeline  0: batched; 1: plain
  resident  queries uploaded beforehand (search_resident) instead of searched from host buffers
  fields    "all": the columns RepeatMasker asks for, alignments included; "short": score and ranges

A pass is one search call and the outfmt-6 text of every HSP; the text is the output, as bytes at
the front of a buffer that the case's sizes give (zeros after it).  Nothing in it is computed in
floating point on the GPU, so there is no 64-bit value to give: the bytes stay what they are.
"""
from __future__ import annotations

import math

import numpy as np

from rmblast_b200 import api, synth, train_sched

FIELDS = {
    "all": ("6 score perc_sub perc_query_gap perc_db_gap qseqid qstart qend qlen sstrand sseqid sstart send slen "
            "kdiv cpg_kdiv transi transv cpg_sites qseq sseq"),
    "short": "6 score perc_sub qseqid qstart qend sseqid sstart send",
}
# Mean consensus length of a library: log-normal (median 1.5 kb), or uniform for a self search.
LIBRARY_MEAN = 2_330
SELF_MEAN = 5_100
# Preliminary-DP cells a search needs per query base and library base, as the reference counts
# them on these workloads, and the integer operations of one cell (three maxima, the additions
# and the X-drop comparison).
CELLS_PER_PAIR_OF_BASES = {7: 3.4e-3, 11: 1.1e-3, 14: 2.5e-4}
OPS_PER_CELL = 11


def _case(name=None, *, queries, bp, library, word=11, spread=0.0, self_search=False, flags="repeatmasker",
          dust=False, schedule=0, pipeline=0, resident=False, fields="all"):
    c = {"queries": queries, "bp": bp, "spread": spread, "library": library, "self": self_search, "word": word,
         "flags": flags, "dust": dust, "schedule": schedule, "pipeline": pipeline, "resident": resident,
         "fields": fields}
    return c if name is None else {"name": name, **c}


def listed():
    return [
        # one short sequence (a new consensus, a clone end) looked up in a library: latency
        _case("one_sequence", queries=1, bp=1_537, library=500),
        # one genome piece of 100 kb against a small library at RepeatMasker's sensitive word size
        _case("genome_100kb_word7", queries=1, bp=100_000, library=50, word=7),
        # RepeatMasker's batch: one 60 kb piece a call, against a full library
        _case("one_60kb_chunk", queries=1, bp=60_000, library=2_000),
        # a bulk search: 60 kb pieces of a genome, many to a call
        _case("chunks_60kb", queries=120, bp=60_000, library=2_000),
        # the same pieces through the plain pipeline
        _case("chunks_60kb_plain", queries=60, bp=60_000, library=2_000, pipeline=1),
        # contigs of a draft assembly, 1-200 kb, from host buffers in arrival order
        _case("contigs", queries=200, bp=20_000, spread=1.0, library=2_000),
        # the benchmark's step: 1,000 contigs resident on the device, learned order
        _case("contigs_bulk_learned", queries=1_000, bp=20_000, spread=1.0, library=2_000, schedule=1, resident=True,
              fields="short"),
        # many short sequences (reads, clone ends) at word 14
        _case("short_sequences_word14", queries=3_000, bp=900, spread=0.5, library=1_000, word=14),
        # a library against itself (redundancy removal, family building), masklevel off
        _case("library_self_search", queries=40, bp=SELF_MEAN, library=1_000, word=7, self_search=True),
        # rmblastn's command-line defaults, DUST on: every word hit's alignment comes out
        _case("defaults_dust", queries=24, bp=30_011, library=200, flags="defaults", dust=True),
        # one contig at RepeatMasker's settings with DUST left on (rmblastn's default)
        _case("contig_150kb_dust", queries=1, bp=150_000, library=50, word=7, dust=True),
        # a long contig: past 1,999,800 bp a query is cut into chunks
        _case("long_contig", queries=1, bp=2_100_000, library=50, word=7),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["single", "single", "fixed", "fixed", "contigs", "contigs", "short", "self", "dust", "long"])
    if kind == "single":
        word = rng.choice([7, 11, 11, 14])
        return _case(queries=1, bp=_log(rng, 200, 120_000), library=_log(rng, 20, 400 if word == 7 else 2_500),
                     word=word, dust=rng.random() < 0.25)
    if kind == "fixed":
        return _case(queries=_log(rng, 2, 150), bp=_log(rng, 5_000, 100_000), library=_log(rng, 100, 2_000),
                     word=rng.choice([11, 11, 14]), pipeline=int(rng.random() < 0.2))
    if kind == "contigs":
        return _case(queries=_log(rng, 5, 600), bp=_log(rng, 8_000, 25_000), spread=rng.uniform(0.4, 1.1),
                     library=_log(rng, 200, 2_000), schedule=rng.choice([0, 1]), resident=rng.random() < 0.5,
                     fields=rng.choice(["all", "short"]))
    if kind == "short":
        return _case(queries=_log(rng, 20, 4_000), bp=_log(rng, 150, 1_500), spread=rng.uniform(0.2, 0.6),
                     library=_log(rng, 100, 1_500), word=rng.choice([11, 14]))
    if kind == "self":
        return _case(queries=_log(rng, 8, 50), bp=SELF_MEAN, library=_log(rng, 150, 1_000), word=7,
                     self_search=True)
    if kind == "dust":
        rm = rng.random() < 0.5
        return _case(queries=_log(rng, 2, 40), bp=_log(rng, 4_000, 60_000 if rm else 30_000),
                     library=_log(rng, 50, 1_000 if rm else 200), flags="repeatmasker" if rm else "defaults", dust=True)
    return _case(queries=1, bp=_log(rng, 200_000, 2_150_000), library=rng.randint(10, 50), word=rng.choice([7, 11]))


def _add_simple_repeats(r, g, frac=0.02):
    """Microsatellites and homopolymer runs (what DUST masks) over `frac` of a sequence."""
    left = frac * len(g)
    while left > 0:
        unit = synth.random_dna(r, int(r.integers(1, 7)))
        n = min(int(r.integers(20, 120)), len(g) // 2)
        pos = int(r.integers(0, len(g) - n))
        g[pos:pos + n] = np.resize(unit, n)
        left -= n
    return g


def _inputs(case, seed):
    """(query ids, queries, library records), all as ASCII sequences."""
    if case["self"]:
        recs, _, _ = synth.workload("allvsall", seed=seed, scale=case["library"] / 5000.0)
        step = max(1, len(recs) // case["queries"])
        qs = recs[::step][:case["queries"]]
        return [n for n, _ in qs], [s for _, s in qs], recs
    rng = np.random.default_rng([seed, 1 << 20])
    n = case["library"]
    lib = synth.library(rng, n, synth.lognormal_lengths(rng, n, 1500.0, 2500.0 * n, 100, 12_000))
    ids, qs = [], []
    for i in range(case["queries"]):
        r = np.random.default_rng([seed, i])
        bp = case["bp"]
        if case["spread"]:
            lo, hi = (60, 4_000) if bp < 2_000 else (1_000, 200_000)
            bp = int(np.clip(np.round(r.lognormal(np.log(bp), case["spread"])), lo, hi))
        g = synth.random_dna(r, bp)
        # a planted copy has at least 50 bases and has to be shorter than the sequence
        fit = [c for c in lib if len(c) < bp] or [c[:max(60, bp // 2)] for c in lib[:16]]
        g = synth.plant(r, g, fit, 0.45, None, (0.02, 0.35), (0.01, 0.05))
        if case["dust"]:
            g = _add_simple_repeats(r, g)
        ids.append(f"seq{i}")
        qs.append(synth.add_n_runs(r, g) if bp >= 5_000 else g)
    return ids, qs, [(f"cons{i}", s) for i, s in enumerate(lib)]


def prepare(case, seed):
    ids, qs, recs = _inputs(case, seed)
    rm = case["flags"] == "repeatmasker"
    flags = synth.RM_FLAGS if rm else synth.DEFAULT_FLAGS
    params = api.SearchParams(word_size=case["word"], complexity_adjust=rm, dust=case["dust"],
                              mask_level=80 if rm and not case["self"] else -1, schedule=case["schedule"],
                              pipeline=case["pipeline"], device=0, **flags)
    matrix = api.ScoreMatrix.from_text(synth.MATRIX_TEXT, synth.MATRIX_NAME)
    searcher = api.Searcher(params, matrix, api.SubjectDb.from_records(recs))
    if case["schedule"]:
        searcher.set_schedule_model(train_sched.load_model())
    queries = [api.encode(q) for q in qs]
    state = {"searcher": searcher, "ids": ids, "queries": queries, "fields": FIELDS[case["fields"]], "resident": None,
             "buffer": np.zeros(_text_capacity(case), dtype=np.uint8), "used": 0}
    if case["resident"]:
        state["resident"] = searcher.upload(queries)
    return state


def run(state):
    s = state["searcher"]
    if state["resident"] is not None:
        res = s.search_resident(state["resident"], state["ids"])
    else:
        res = s.search(state["queries"], state["ids"])
    text = np.frombuffer(res.tabular(state["fields"]).encode(), dtype=np.uint8)
    buf, n = state["buffer"], len(text)
    buf[:n] = text
    buf[n:state["used"]] = 0
    state["used"] = n
    return {"tabular": buf}


def exact(case, seed):
    return None


def _bases(case):
    return case["queries"] * case["bp"] * math.exp(case["spread"] ** 2 / 2)


def _library_bases(case):
    return case["library"] * (SELF_MEAN if case["self"] else LIBRARY_MEAN)


def _text_capacity(case):
    """Bytes of the output buffer, past what the text of such a case comes to: about one byte a
    query base with the alignments, three in a self search; with the defaults' cutoff of 0 every
    word hit prints a line (5.5e-5 bytes a pair of bases)."""
    q = _bases(case)
    per_hit = 1.5e-4 * q * _library_bases(case) if case["flags"] == "defaults" else 0
    return (1 << 17) + int((12 if case["self"] else 3) * q + per_hit)


def work(case):
    """Bytes: the queries and the packed library read once, the text written once (the alignments
    of the planted 45% of the query bases, both rows).  Operations: the preliminary DP's cells."""
    q, lib = _bases(case), _library_bases(case)
    text = 0.9 * q if case["fields"] == "all" else 0.03 * q
    return {"bytes": q + lib / 4 + text, "flops": CELLS_PER_PAIR_OF_BASES[case["word"]] * q * lib * OPS_PER_CELL}
