"""Tracebacks with scores up to and past what the register-band kernel's dead cells allow (255), against the
oracle's: extensions that begin with mismatches beside cheap gaps and a small X-drop, so that a threshold
stays near its start while off-diagonal matches add the largest scores."""
import numpy as np
import pytest

import oracle_ref as O
from rmblast_b200 import api, synth


def matrix_text(top):
    a, ts, tv, n = round(0.9 * top), -round(0.8 * top), -round(1.5 * top), -max(1, top // 10)
    rows = [("A", (a, tv, ts, tv, n)), ("C", (tv, top, tv, ts, n)), ("G", (ts, tv, top, tv, n)), ("T", (tv, ts, tv, a, n)),
            ("N", (n,) * 5)]
    return ("# FREQS A 0.295 C 0.205 G 0.205 T 0.295\n  A C G T N\n" +
            "".join(f"{b} {' '.join(map(str, v))}\n" for b, v in rows))


def sequences(rng):
    lib = [synth.random_dna(rng, int(k)) for k in rng.integers(150, 700, 7)]
    qs = []
    for i in range(9):
        c = lib[int(rng.integers(len(lib)))]
        c = c if i % 2 else synth.revcomp(c)
        qs.append(np.concatenate([synth.random_dna(rng, int(rng.integers(0, 80))),
                                  synth.mutate(rng, c, float(rng.uniform(0.15, 0.4)), float(rng.uniform(0, 0.05))),
                                  synth.random_dna(rng, int(rng.integers(0, 80)))]))
    return qs, lib


@pytest.mark.gpu
@pytest.mark.parametrize("gaps", [(20, 1, 0), (5, 2, 30), (0, 5, 0), (40, 40, 700)])
@pytest.mark.parametrize("top", [127, 255, 256, 340, 600, 2000])
def test_tracebacks_match_the_oracle(top, gaps):
    """top: the matrix's largest score; gaps: gap open, gap extend, final X-drop."""
    rng = np.random.default_rng([0x5C0E, top, *gaps])
    qs, lib = sequences(rng)
    text = matrix_text(top)
    p = dict(gap_open=gaps[0], gap_extend=gaps[1], word_size=5, xdrop_ungap=2 * top, xdrop_gap=gaps[0] + gaps[1],
             xdrop_gap_final=gaps[2], min_raw_gapped_score=6 * top, complexity_adjust=1, dust=0, mask_level=101)
    qf = synth.to_fasta([f"q{i}" for i in range(len(qs))], qs)
    dbf = synth.to_fasta([f"s{i}" for i in range(len(lib))], lib)
    sp = api.SearchParams(**dict(p, complexity_adjust=True, dust=False))
    s = api.Searcher(sp, api.ScoreMatrix.from_text(text, "scaled"), api.SubjectDb.from_fasta(dbf))
    recs = api.read_fasta(qf)
    enc = [api.encode(x) for _, x in recs]
    want = O.stage_text(qf, dbf, text, "scaled", p, 4)
    assert len(want) > 500
    assert np.array_equal(s.stage(enc, 4), want)
    lines, _, _ = O.search_text(qf, dbf, text, "scaled", p, O.RM_FIELDS)
    assert s.search(enc, [n for n, _ in recs]).tabular(O.RM_FIELDS) == lines
