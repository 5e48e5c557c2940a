"""The packed-row preliminary DP against the warp kernel (kernels=1), which the oracle tests pin:
the same prelim records, the same DP cells, the same output."""
import numpy as np
import pytest

from rmblast_b200 import api, synth

FIELDS = "6 score perc_sub qseqid qstart qend sseqid sstart send qseq sseq"


def sequences(rng, n_lib, n_query):
    """Consensi, and queries of mutated copies (many short indels, so the alignment's diagonal
    drifts both ways), exact copies longer than the score range of a 16-bit value, N and other
    ambiguity codes, and sequences only a few bases longer than the word."""
    lib = [synth.random_dna(rng, int(k)) for k in rng.integers(60, 2500, n_lib)] + [synth.random_dna(rng, 9000)]
    qs = []
    for i in range(n_query):
        parts = []
        for _ in range(int(rng.integers(1, 6))):
            c = lib[int(rng.integers(len(lib)))]
            c = c if rng.random() < 0.5 else synth.revcomp(c)
            s = int(rng.integers(0, len(c) - 20))
            frag = synth.mutate(rng, c[s:s + int(rng.integers(20, 3000))], float(rng.uniform(0, 0.35)),
                                float(rng.uniform(0, 0.12)))
            parts += [synth.random_dna(rng, int(rng.integers(1, 200))), frag]
        g = np.concatenate(parts)
        kind = i % 4
        if kind == 1:
            g[rng.integers(0, len(g), len(g) // 50 + 1)] = ord("N")
        elif kind == 2:
            g[rng.integers(0, len(g), len(g) // 80 + 1)] = rng.choice(np.frombuffer(b"RYMKWSBDHV", np.uint8))
        qs.append(g)
    qs += [lib[-1].copy(), synth.revcomp(lib[-1])]
    qs += [lib[0][:k].copy() for k in (7, 8, 9, 11, 12, 15, 31, 32, 33, 47, 48, 49, 60)]
    qs += [np.concatenate([lib[1][:40], lib[1][52:]]), np.concatenate([lib[1][:30], lib[0][:14], lib[1][30:]])]
    return qs, lib


@pytest.mark.gpu
@pytest.mark.parametrize("pipeline", [0, 1])
@pytest.mark.parametrize("gaps", [(20, 5, 100, 150), (20, 5, 30, 150), (12, 4, 76, 150), (28, 5, 108, 150),
                                  (25, 8, 128, 150), (20, 5, 128, 150), (20, 5, 100, 60), (20, 5, 30, 0)])
def test_packed_rows_match_the_warp_kernel(gaps, pipeline):
    """gaps: gap open, gap extend, X-drop, gapped cutoff; a cutoff at or under a word hit's score (70)
    takes every record to k_prelim_pack, one above it k_prelim_dual first."""
    rng = np.random.default_rng([0x9ACC, *gaps[:3]])
    qs, lib = sequences(rng, 40, 60)
    db = api.SubjectDb.from_records([(f"s{i}", s) for i, s in enumerate(lib)])
    m = api.ScoreMatrix.from_text(synth.MATRIX_TEXT, synth.MATRIX_NAME)
    enc = [api.encode(q) for q in qs]
    got = []
    for kernels in (0, 1):
        s = api.Searcher(api.SearchParams(gap_open=gaps[0], gap_extend=gaps[1], word_size=7, xdrop_ungap=400,
                                          xdrop_gap=gaps[2], xdrop_gap_final=200, min_raw_gapped_score=gaps[3],
                                          complexity_adjust=True, kernels=kernels, pipeline=pipeline), m, db)
        pre = s.stage(enc, 2)
        res = s.search(enc)
        got.append((pre[np.lexsort(pre.T[::-1])], res.counters["so_cells"], res.counters["prelims"],
                    res.tabular(FIELDS)))
    assert len(got[0][0]) > 100
    assert np.array_equal(got[0][0], got[1][0])
    assert got[0][1:] == got[1][1:]


@pytest.mark.gpu
@pytest.mark.parametrize("gaps", [(20, 5, 100, 150), (20, 55, 128, 150)])
def test_many_records_a_thread(gaps):
    """Millions of random word hits: each half of a k_prelim_dual thread runs tens of records one after the
    other (their values climb until they are moved down), also at nearly the steepest gap it takes."""
    rng = np.random.default_rng([0x9ACD, *gaps[:3]])
    lib = [synth.random_dna(rng, int(k)) for k in rng.integers(60, 6000, 60)]
    qs = [synth.plant(rng, synth.random_dna(rng, n), lib, 0.05, None, (0.05, 0.3), (0.01, 0.05)) for n in (250_000, 60_000)]
    db = api.SubjectDb.from_records([(f"s{i}", s) for i, s in enumerate(lib)])
    m = api.ScoreMatrix.from_text(synth.MATRIX_TEXT, synth.MATRIX_NAME)
    enc = [api.encode(q) for q in qs]
    got = []
    for kernels in (0, 1):
        s = api.Searcher(api.SearchParams(gap_open=gaps[0], gap_extend=gaps[1], word_size=7, xdrop_ungap=400,
                                          xdrop_gap=gaps[2], xdrop_gap_final=200, min_raw_gapped_score=gaps[3],
                                          complexity_adjust=True, kernels=kernels), m, db)
        res = s.search(enc)
        got.append((res.counters["so_cells"], res.counters["prelims"], res.counters["ungapped"], res.tabular(FIELDS)))
    assert got[0][2] > 10 * 148 * 3 * 128 * 2  # halves of 12 warps on each of 148 SMs
    assert got[0] == got[1]
