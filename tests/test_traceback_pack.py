"""The register-band traceback against the oracle's: boxes, scores and edit scripts on alignments that
drift across its window (long and many indels both ways), outgrow it, and meet N and other ambiguity
codes in the query and in the library."""
import numpy as np
import pytest

import oracle_ref as O
from rmblast_b200 import api, synth


def sequences(rng):
    lib = [synth.random_dna(rng, int(k)) for k in rng.integers(80, 1500, 8)] + [synth.random_dna(rng, 5000)]
    qs = []
    for i in range(14):
        c = lib[int(rng.integers(len(lib)))]
        c = c if rng.random() < 0.5 else synth.revcomp(c)
        frag = synth.mutate(rng, c, float(rng.uniform(0, 0.25)), float(rng.uniform(0, 0.08)))
        if i % 3 == 0 and len(frag) > 200:  # deletions or insertions of up to 40 bases, one way
            at = np.sort(rng.integers(50, len(frag) - 50, 6))
            parts, prev = [], 0
            for p in at:
                if p < prev:
                    continue
                parts.append(frag[prev:p])
                k = int(rng.integers(5, 41))
                if i % 2:
                    prev = p + k
                else:
                    parts.append(synth.random_dna(rng, k))
                    prev = p
            frag = np.concatenate(parts + [frag[prev:]])
        g = np.concatenate([synth.random_dna(rng, int(rng.integers(1, 60))), frag, synth.random_dna(rng, int(rng.integers(0, 60)))])
        if i % 4 == 1:
            g[rng.integers(0, len(g), len(g) // 60 + 1)] = ord("N")
        elif i % 4 == 2:
            g[rng.integers(0, len(g), len(g) // 90 + 1)] = rng.choice(np.frombuffer(b"RYMKWSBDHV", np.uint8))
        qs.append(g)
    for i in (1, 3):  # ambiguity codes in the library
        lib[i][rng.integers(0, len(lib[i]), len(lib[i]) // 40)] = ord("N")
    lib[5][rng.integers(0, len(lib[5]), len(lib[5]) // 40)] = ord("R")
    qs += [lib[-1].copy(), lib[0][:30].copy()]
    return qs, lib


@pytest.mark.gpu
@pytest.mark.parametrize("pipeline", [0, 1])
@pytest.mark.parametrize("gaps", [(20, 5, 200), (20, 5, 100), (12, 4, 150), (25, 8, 250), (20, 5, 300), (20, 5, 400)])
def test_tracebacks_match_the_oracle(gaps, pipeline):
    """gaps: gap open, gap extend, final X-drop; at 300 the initial row nearly fills the window, 400 is past
    what the register-band kernel takes."""
    rng = np.random.default_rng([0x7BAC, *gaps])
    qs, lib = sequences(rng)
    p = dict(O.RM_PARAMS, gap_open=gaps[0], gap_extend=gaps[1], xdrop_gap_final=gaps[2], word_size=8,
             complexity_adjust=1, dust=0, mask_level=101)
    qf = synth.to_fasta([f"q{i}" for i in range(len(qs))], qs)
    dbf = synth.to_fasta([f"s{i}" for i in range(len(lib))], lib)
    sp = api.SearchParams(gap_open=gaps[0], gap_extend=gaps[1], word_size=8, xdrop_ungap=p["xdrop_ungap"],
                          xdrop_gap=p["xdrop_gap"], xdrop_gap_final=gaps[2],
                          min_raw_gapped_score=p["min_raw_gapped_score"], complexity_adjust=True, mask_level=101,
                          pipeline=pipeline)
    s = api.Searcher(sp, api.ScoreMatrix.from_text(synth.MATRIX_TEXT, synth.MATRIX_NAME), api.SubjectDb.from_fasta(dbf))
    recs = api.read_fasta(qf)
    enc = [api.encode(x) for _, x in recs]
    got = s.stage(enc, 4)
    want = O.stage_text(qf, dbf, synth.MATRIX_TEXT, synth.MATRIX_NAME, p, 4)
    assert len(want) > 10
    assert np.array_equal(got, want)
    text, _, _ = O.search_text(qf, dbf, synth.MATRIX_TEXT, synth.MATRIX_NAME, p, O.RM_FIELDS)
    assert s.search(enc, [n for n, _ in recs]).tabular(O.RM_FIELDS) == text
