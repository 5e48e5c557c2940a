"""Word hits of the scan, in order, against the oracle's: subjects around the edges of a round of 128 scan
positions, whole pairs and stretches of them, dense cells and pairs of more hits than a warp's stage holds."""
import numpy as np
import pytest

import oracle_ref as O
from rmblast_b200 import api, synth


def workload(case, word, rng):
    if case == "edges":  # 1 to 3 rounds and one position either way, at every stride a word size takes
        lens = sorted({max(word, (word - lw + 1) * (128 * r + d) + lw + e)
                       for lw in (min(word, 8), min(word, 11)) for r in (0, 1, 3) for d in (-1, 0, 1) for e in (-1, 0)})
        lib = [synth.random_dna(rng, n) for n in lens]
        qs = [synth.plant(rng, synth.random_dna(rng, n), lib, 0.4, None, (0.0, 0.1), (0.0, 0.02)) for n in (2_000, 30_000)]
    elif case == "pairs":  # more pairs than the chip has warps: one unit a pair
        lib = [synth.random_dna(rng, int(n)) for n in rng.integers(60, 1500, 420)]
        qs = [synth.plant(rng, synth.random_dna(rng, int(n)), lib, 0.4, None, (0.02, 0.2), (0.01, 0.03))
              for n in rng.integers(300, 7000, 60)]
    else:  # "dense": repeats whose words fill one lookup cell, tens of thousands of hits a pair
        unit = synth.random_dna(rng, 31)
        tandem = synth.mutate(rng, np.resize(unit, 6_000), 0.02, 0.0)
        lib = [tandem, synth.random_dna(rng, 9_000), np.resize(np.frombuffer(b"AC", np.uint8), 700)]
        qs = [np.concatenate([synth.random_dna(rng, 500), synth.revcomp(tandem), lib[1][:4_000], lib[2]])]
    qs[0][rng.integers(0, len(qs[0]), 9)] = ord("N")
    lib[-1][rng.integers(0, len(lib[-1]), 3)] = ord("N")
    return qs, lib


@pytest.mark.gpu
@pytest.mark.parametrize("pipeline", [0, 1])
@pytest.mark.parametrize("case,word", [("edges", 7), ("edges", 8), ("edges", 11), ("edges", 14), ("edges", 16),
                                       ("pairs", 11), ("pairs", 14), ("dense", 7), ("dense", 11)])
def test_word_hits_match_the_oracle(case, word, pipeline):
    rng = np.random.default_rng([0x5CA, word, len(case)])
    qs, lib = workload(case, word, rng)
    qf = synth.to_fasta([f"q{i}" for i in range(len(qs))], qs)
    dbf = synth.to_fasta([f"s{i}" for i in range(len(lib))], lib)
    p = dict(O.RM_PARAMS, word_size=word, complexity_adjust=1, dust=0)
    s = api.Searcher(api.SearchParams(word_size=word, complexity_adjust=True, pipeline=pipeline, **synth.RM_FLAGS),
                     api.ScoreMatrix.from_text(synth.MATRIX_TEXT, synth.MATRIX_NAME), api.SubjectDb.from_fasta(dbf))
    got = s.stage([api.encode(x) for _, x in api.read_fasta(qf)], 0)
    want = O.stage_text(qf, dbf, synth.MATRIX_TEXT, synth.MATRIX_NAME, p, 0)
    assert len(want) > 50
    assert np.array_equal(got, want)
