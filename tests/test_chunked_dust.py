"""DUST on queries that are cut into chunks (1,999,800 bp and more), against the oracle, each search several times:
the chunks' masked bytes and their reverse complements are in place before the tables are built."""
import numpy as np
import pytest

import oracle_ref as O
from rmblast_b200 import api, synth


def query(rng, n, lib):
    g = synth.add_n_runs(rng, synth.plant(rng, synth.random_dna(rng, n), lib, 0.2, None, (0.02, 0.3), (0.01, 0.05)))
    # microsatellites of two bases and more (a homopolymer beside an N takes the sequential pass, seconds a query)
    for _ in range(n // 8000):
        k, p = int(rng.integers(20, 300)), int(rng.integers(0, n - 300))
        g[p:p + k] = np.resize(np.concatenate([synth.BASES[:2], synth.random_dna(rng, int(rng.integers(0, 5)))]), k)
    return g


@pytest.mark.gpu
@pytest.mark.parametrize("sizes", [(1_999_800,), (2_310_007, 9_001), (2_000_003, 3_100_001)])
def test_searches_match_the_oracle(sizes):
    rng = np.random.default_rng([0xC4D, len(sizes), sizes[0]])
    lib = [synth.random_dna(rng, int(k)) for k in rng.integers(300, 2500, 8)]
    names = [f"q{i}" for i in range(len(sizes))]
    qs = [query(rng, n, lib) for n in sizes]
    p = dict(O.RM_PARAMS, word_size=11, complexity_adjust=1, dust=1, mask_level=80)
    qf = synth.to_fasta(names, qs)
    dbf = synth.to_fasta([f"s{i}" for i in range(len(lib))], lib)
    want, _, _ = O.search_text(qf, dbf, synth.MATRIX_TEXT, synth.MATRIX_NAME, p, O.RM_FIELDS)
    assert want.count("\n") > 100
    s = api.Searcher(api.SearchParams(**dict(p, complexity_adjust=True, dust=True)),
                     api.ScoreMatrix.from_text(synth.MATRIX_TEXT, synth.MATRIX_NAME), api.SubjectDb.from_fasta(dbf))
    enc = [api.encode(q) for q in qs]
    rq = s.upload(enc)
    for _ in range(4):
        assert s.search(enc, names).tabular(O.RM_FIELDS) == want
        assert s.search_resident(rq, names).tabular(O.RM_FIELDS) == want
    rq.free()
