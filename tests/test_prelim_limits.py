"""The packed-row preliminary DP at the limits of its number ranges: the largest scores and gap extensions
that it takes, an X-drop of 128, alignments of 9,000 bases that stay under the cutoff (so that k_prelim_dual
moves its origin again and again); against the warp kernel (kernels=1), which the oracle tests pin."""
import numpy as np
import pytest

from rmblast_b200 import api, synth
from test_prelim_pack import FIELDS, sequences
from test_traceback_scores import matrix_text


@pytest.mark.gpu
@pytest.mark.parametrize("words_to_cutoff", [0.5, 1.5, 10**5])
@pytest.mark.parametrize("limits", [(125, 112, 1), (117, 53, 5), (47, 60, 40), (1, 65, 63)])
def test_limits_match_the_warp_kernel(limits, words_to_cutoff):
    """limits: the matrix's largest score, gap open, gap extend; words_to_cutoff: the gapped cutoff in word hits
    (under one k_prelim_pack takes every record, over it k_prelim_dual first)."""
    top, go, ge = limits
    rng = np.random.default_rng([0x11A1, *limits])
    qs, lib = sequences(rng, 25, 40)
    db = api.SubjectDb.from_records([(f"s{i}", s) for i, s in enumerate(lib)])
    m = api.ScoreMatrix.from_text(matrix_text(top), "limits")
    enc = [api.encode(q[~np.isin(q, np.frombuffer(b"RYMKWSBDHV", np.uint8))]) for q in qs]
    got = []
    for kernels in (0, 1):
        s = api.Searcher(api.SearchParams(gap_open=go, gap_extend=ge, word_size=7, xdrop_ungap=20 * top, xdrop_gap=128,
                                          xdrop_gap_final=250, min_raw_gapped_score=int(7 * top * words_to_cutoff),
                                          ungapped_cutoff=7 * top, complexity_adjust=True, kernels=kernels), m, db)
        pre = s.stage(enc, 2)
        res = s.search(enc)
        got.append((pre[np.lexsort(pre.T[::-1])], res.counters["so_cells"], res.counters["prelims"],
                    res.tabular(FIELDS)))
    assert got[0][1] > 10**6 and (len(got[0][0]) > 100 or words_to_cutoff > 2)
    assert np.array_equal(got[0][0], got[1][0])
    assert got[0][1:] == got[1][1:]
