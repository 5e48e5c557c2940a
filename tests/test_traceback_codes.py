"""The register-band traceback on libraries with every ambiguity code, whose scores its code table has no room
for, against the oracle's: single codes that enter and leave the window, and windows full of them."""
import numpy as np
import pytest

import oracle_ref as O
from rmblast_b200 import api, synth
from test_traceback_pack import sequences


@pytest.mark.gpu
@pytest.mark.parametrize("pipeline", [0, 1])
@pytest.mark.parametrize("density", [0.002, 0.02, 0.2])
def test_tracebacks_match_the_oracle(density, pipeline):
    rng = np.random.default_rng([0xC0DE, int(1000 * density)])
    qs, lib = sequences(rng)
    for s in lib:
        at = rng.random(len(s)) < density
        s[at] = rng.choice(np.frombuffer(b"RYMKWSBDHVN", np.uint8), int(at.sum()))
    text = (O.GOLDEN / "comparison.matrix").read_text()
    p = dict(O.RM_PARAMS, word_size=8, complexity_adjust=1, dust=0, mask_level=101, min_raw_gapped_score=90)
    qf = synth.to_fasta([f"q{i}" for i in range(len(qs))], qs)
    dbf = synth.to_fasta([f"s{i}" for i in range(len(lib))], lib)
    s = api.Searcher(api.SearchParams(**dict(p, complexity_adjust=True, dust=False), pipeline=pipeline),
                     api.ScoreMatrix.from_text(text, "comparison.matrix"), api.SubjectDb.from_fasta(dbf))
    recs = api.read_fasta(qf)
    enc = [api.encode(x) for _, x in recs]
    want = O.stage_text(qf, dbf, text, "comparison.matrix", p, 4)
    assert len(want) > 10
    assert np.array_equal(s.stage(enc, 4), want)
    lines, _, _ = O.search_text(qf, dbf, text, "comparison.matrix", p, O.RM_FIELDS)
    assert s.search(enc, [n for n, _ in recs]).tabular(O.RM_FIELDS) == lines
