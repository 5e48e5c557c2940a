"""The preliminary DP around the lines where a query set's ambiguity codes other than N take it from the packed
rows to the thread-per-extension kernel (one 32-base stretch in 200 with such a code, and many records):
none, a few, at the line, over it, many; against the warp kernel (kernels=1), which the oracle tests pin."""
import numpy as np
import pytest

from rmblast_b200 import api, synth, train_sched
from test_prelim_pack import FIELDS, sequences

LINE = 200  # 32-base stretches to each one with such a code


def with_codes(rng, qs, stretches):
    """The queries with N for their ambiguity codes, and codes other than N in so many 32-base stretches."""
    out = []
    for q in qs:
        q = q.copy()
        q[~np.isin(q, np.frombuffer(b"ACGT", np.uint8))] = ord("N")
        out.append(q)
    places = [(i, j) for i, q in enumerate(out) for j in range(0, len(q), 32)]
    for k in rng.permutation(len(places))[:stretches]:
        i, j = places[k]
        width = min(32, len(out[i]) - j)
        at = j + rng.integers(0, width, int(rng.integers(1, 4)))
        out[i][at] = rng.choice(np.frombuffer(b"RYMKWSBDHV", np.uint8), len(at))
    return out


@pytest.mark.gpu
@pytest.mark.parametrize("sparse,pipeline,schedule", [(True, 0, 0), (True, 0, 1), (True, 0, 2), (False, 0, 0), (False, 1, 0)])
@pytest.mark.parametrize("part", [0.0, 0.2, 1.0, 1.8, 20.0])
@pytest.mark.parametrize("gaps", [(20, 5, 100, 150), (25, 8, 128, 60)])
def test_codes_match_the_warp_kernel(gaps, part, sparse, pipeline, schedule):
    """gaps: gap open, gap extend, X-drop, gapped cutoff; part: of the stretches that the line lies at; sparse:
    every word hit counts as a record to come (else a part of them, or the records themselves)."""
    rng = np.random.default_rng([0x0DD5, *gaps[:3]])
    qs, lib = sequences(rng, 25, 80)
    bases = sum(len(q) + 2 for q in qs)
    qs = with_codes(rng, qs, int(part * bases / 32 / LINE))
    db = api.SubjectDb.from_records([(f"s{i}", s) for i, s in enumerate(lib)])
    m = api.ScoreMatrix.from_text(synth.MATRIX_TEXT, synth.MATRIX_NAME)
    enc = [api.encode(q) for q in qs]
    got = []
    for kernels in (0, 1):
        s = api.Searcher(api.SearchParams(gap_open=gaps[0], gap_extend=gaps[1], word_size=7, xdrop_ungap=400,
                                          xdrop_gap=gaps[2], xdrop_gap_final=200, min_raw_gapped_score=gaps[3],
                                          complexity_adjust=True, kernels=kernels, pipeline=pipeline,
                                          schedule=schedule if kernels == 0 else 0), m, db)
        if kernels == 0 and schedule:
            s.set_schedule_model(train_sched.load_model())
        if sparse:
            s.set_tune(dict(s.tune(), dedup_extend_hits_per_pair=-1))
        pre = s.stage(enc, 2)
        res = s.search(enc)
        got.append((pre[np.lexsort(pre.T[::-1])], res.counters["so_cells"], res.counters["prelims"],
                    res.tabular(FIELDS)))
        assert not sparse or part <= 1 or part / LINE * res.counters["word_hits"] > 7500
    assert len(got[0][0]) > 100
    assert np.array_equal(got[0][0], got[1][0])
    assert got[0][1:] == got[1][1:]
