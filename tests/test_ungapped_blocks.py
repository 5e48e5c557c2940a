"""Ungapped extensions, eight bases a step, against the oracle's: sequences that end within a step of
the word hit, every alignment of the two sequences' words, ambiguity codes, both strands."""
import numpy as np
import pytest

import oracle_ref as O
from rmblast_b200 import api, synth


@pytest.mark.gpu
@pytest.mark.parametrize("pipeline", [0, 1])
@pytest.mark.parametrize("xdrop", [1, 40, 400])
def test_ungapped_hits_match_the_oracle(xdrop, pipeline):
    rng = np.random.default_rng([0x0B10, xdrop])
    lib = [synth.random_dna(rng, n) for n in list(range(8, 42)) + [300, 1000, 1001, 1002, 1003]]
    qs = []
    for i, s in enumerate(lib):
        a, b = rng.integers(0, 20, 2)
        core = s if i % 2 else synth.revcomp(s)
        g = np.concatenate([synth.random_dna(rng, int(a)), synth.mutate(rng, core, 0.06, 0.0), synth.random_dna(rng, int(b))])
        if i % 5 == 4:
            g[rng.integers(0, len(g), 2)] = rng.choice(np.frombuffer(b"NRYKM", np.uint8), 2)
        qs += [core[:int(rng.integers(8, len(core) + 1))].copy(), g]
    qf = synth.to_fasta([f"q{i}" for i in range(len(qs))], qs)
    dbf = synth.to_fasta([f"s{i}" for i in range(len(lib))], lib)
    p = dict(O.RM_PARAMS, word_size=7, complexity_adjust=1, dust=0, xdrop_ungap=xdrop)
    s = api.Searcher(api.SearchParams(word_size=7, complexity_adjust=True, pipeline=pipeline,
                                      **dict(synth.RM_FLAGS, xdrop_ungap=xdrop)),
                     api.ScoreMatrix.from_text(synth.MATRIX_TEXT, synth.MATRIX_NAME), api.SubjectDb.from_fasta(dbf))
    got = s.stage([api.encode(x) for _, x in api.read_fasta(qf)], 1)
    want = O.stage_text(qf, dbf, synth.MATRIX_TEXT, synth.MATRIX_NAME, p, 1)
    assert len(want) > 100
    assert np.array_equal(got, want)
