"""The bucket-parallel diagonal dedup against the plain pipeline's (a pair a thread, every hit
extended first), which the oracle tests pin: the same seeds, ungapped records and output."""
import numpy as np
import pytest

from rmblast_b200 import api, synth

FIELDS = "6 score perc_sub qseqid qstart qend sseqid sstart send qseq sseq"


def workload(case, rng):
    if case == "sparse":  # many pairs, few hits a pair: runs of one hit
        lib = [synth.random_dna(rng, int(k)) for k in rng.integers(60, 3000, 300)]
        qs = [synth.plant(rng, synth.random_dna(rng, 4000), lib, 0.4, None, (0.02, 0.3), (0.01, 0.05)) for _ in range(12)]
        return qs, lib, 11
    if case == "dense":  # few pairs of tens of thousands of hits, both strands
        lib = [synth.random_dna(rng, int(k)) for k in (3000, 2500, 90, 4000)]
        q = synth.plant(rng, synth.random_dna(rng, 90_000), lib, 0.4, None, (0.02, 0.3), (0.01, 0.05))
        return [q, synth.revcomp(q)[:70_000]], lib, 7
    # long identical diagonals and tandem repeats: runs of thousands of hits, chains of several cells
    a = synth.random_dna(rng, 30_000)
    unit = synth.random_dna(rng, 23)
    tandem = synth.mutate(rng, np.resize(unit, 6000), 0.05, 0.01)
    lib = [a[5000:25_000].copy(), synth.revcomp(a[:12_000]), np.concatenate([tandem, a[:3000]])]
    return [a, np.concatenate([a[2000:9000], tandem, synth.mutate(rng, a[9000:20_000], 0.1, 0.02)])], lib, 7


@pytest.mark.gpu
@pytest.mark.parametrize("case", ["sparse", "dense", "identical"])
def test_bucket_replay_matches_the_pair_replay(case):
    rng = np.random.default_rng([0xB0C, len(case)])
    qs, lib, ws = workload(case, rng)
    enc = [api.encode(q) for q in qs]
    db = api.SubjectDb.from_records([(f"s{i}", s) for i, s in enumerate(lib)])
    m = api.ScoreMatrix.from_text(synth.MATRIX_TEXT, synth.MATRIX_NAME)
    got = []
    for pipeline in (0, 1):
        s = api.Searcher(api.SearchParams(word_size=ws, complexity_adjust=True, pipeline=pipeline, **synth.RM_FLAGS), m, db)
        res = s.search(enc)
        c = res.counters
        got.append((res.tabular(FIELDS), *(c[k] for k in ("word_hits", "ungapped", "prelim_dp", "prelims", "so_cells"))))
        if pipeline == 0 and case == "dense":
            assert c["word_hits"] >= 8192 * len(qs) * len(lib)  # the range takes the leaders' path
        # without the extension of admitted hits only, the replay of all hits extended first
        s.set_tune({"dedup_extend_hits_per_pair": -1})
        got.append((s.search(enc).tabular(FIELDS), *got[-1][1:]))
    assert got[0][2] > 100
    assert all(g == got[0] for g in got[1:])
