"""The launch knobs of the thread-per-extension DP with parameters that the packed rows do not take (an X-drop
over 128; an initial row wider than their window), so that its other group sizes, grids and cell budgets run:
the oracle's text and the default shape's cells for each, in the graph, stage by stage and plain."""
import pytest

import oracle_ref as O
from rmblast_b200 import api, synth
from test_gpu_parity import FIELDS, searcher, synthetic

GAPS = [(20, 5, 150), (25, 3, 120)]  # gap open, gap extend, preliminary X-drop


def case(gaps, name, scale):
    qf, dbf, p = synthetic(name, scale, synth.RM_FLAGS)
    p = dict(p, gap_open=gaps[0], gap_extend=gaps[1], xdrop_gap=gaps[2])
    want, _, _ = O.search_text(qf, dbf, synth.MATRIX_TEXT, synth.MATRIX_NAME, p, FIELDS, threads=16)
    assert want.count("\n") > 20
    recs = api.read_fasta(qf)
    return dbf, p, want, [api.encode(x) for _, x in recs], [n for n, _ in recs]


@pytest.mark.gpu
@pytest.mark.parametrize("gaps", GAPS)
@pytest.mark.parametrize("name,scale", [("plain", 0.005), ("allvsall", 0.02)])
def test_knobs_leave_output_unchanged(name, scale, gaps):
    dbf, p, want, enc, ids = case(gaps, name, scale)
    s = searcher(p, synth.MATRIX_TEXT, synth.MATRIX_NAME, dbf)
    default = s.tune()
    res = s.search(enc, ids)
    assert res.tabular(FIELDS) == want
    cells = res.counters["so_cells"]
    for graph in (1, 0, 2):
        for knobs in (dict(prelim_group=4), dict(prelim_group=16), dict(prelim_budget_div=16), dict(prelim_budget_div=4096),
                      dict(prelim_blocks_per_sm=1), dict(prelim_window=16, prelim_group=4, prelim_budget_div=4096)):
            s.set_tune(dict(default, graph=graph, **knobs))
            res = s.search(enc, ids)
            assert res.tabular(FIELDS) == want, (graph, knobs)
            assert res.counters["so_cells"] == cells, (graph, knobs)
    s.set_tune(default)
    r = s.autotune(enc[:max(1, len(enc) // 2)])
    assert r["best_ms"] <= r["default_ms"] and r["tune"] == s.tune()
    assert s.search(enc, ids).tabular(FIELDS) == want


@pytest.mark.gpu
@pytest.mark.parametrize("gaps", GAPS)
def test_plain_pipeline_matches_the_oracle(gaps):
    dbf, p, want, enc, ids = case(gaps, "plain", 0.005)
    assert searcher(p, synth.MATRIX_TEXT, synth.MATRIX_NAME, dbf, pipeline=1).search(enc, ids).tabular(FIELDS) == want


@pytest.mark.gpu
@pytest.mark.parametrize("name,scale", [("plain", 0.01), ("allvsall", 0.03)])
def test_autotune_leaves_knobs_that_reach_no_launch(name, scale):
    """Where the packed rows take every record, the thread-per-extension DP's knobs stay at their defaults."""
    qf, dbf, p = synthetic(name, scale, synth.RM_FLAGS)
    s = searcher(p, synth.MATRIX_TEXT, synth.MATRIX_NAME, dbf)
    default = s.tune()
    enc = [api.encode(x) for _, x in api.read_fasta(qf)]
    for _ in range(3):
        r = s.autotune(enc)
        assert r["tune"] == s.tune() and r["best_ms"] <= r["default_ms"]
        for k in ("prelim_group", "prelim_blocks_per_sm", "prelim_budget_div"):
            assert s.tune()[k] == default[k], k
