"""The packed DP's copy of the library (three bytes a base): made only for parameters that use it, and whole."""
import numpy as np
import pytest

from rmblast_b200 import api, synth


@pytest.mark.gpu
def test_copy_only_where_it_is_used():
    import torch
    rng = np.random.default_rng(0x11B)
    db = api.SubjectDb.from_records([(f"s{i}", synth.random_dna(rng, 4_000_000)) for i in range(16)])
    m = api.ScoreMatrix.from_text(synth.MATRIX_TEXT, synth.MATRIX_NAME)
    torch.cuda.init()
    used = {}
    for name, kw in (("warm", {}), ("packed", {}), ("x150", dict(xdrop_gap=150)), ("warp", dict(kernels=1))):
        torch.cuda.synchronize()
        before = torch.cuda.mem_get_info()[0]
        s = api.Searcher(api.SearchParams(**dict(synth.RM_FLAGS, word_size=11, **kw)), m, db)
        torch.cuda.synchronize()
        used[name] = before - torch.cuda.mem_get_info()[0]
        s.close()
    copy = 3 * db.total_letters()
    assert used["packed"] - used["warp"] > 0.9 * copy
    assert abs(used["x150"] - used["warp"]) < 0.1 * copy


@pytest.mark.gpu
@pytest.mark.parametrize("length", [4_095, 300_007, 1_200_001])
def test_copies_of_long_subjects(length):
    """Several blocks copy a long subject: records, cells and text as the warp kernel's (kernels=1), which has no copy."""
    rng = np.random.default_rng([0x11B, length])
    chrom = synth.random_dna(rng, length)
    lib = [("short", synth.random_dna(rng, 50)), ("long", chrom), ("last", synth.random_dna(rng, 777))]
    qs = [synth.mutate(rng, chrom[p:p + 900] if i % 2 else synth.revcomp(chrom[p:p + 900]), 0.1, 0.02)
          for i, p in enumerate([0, length // 3, 2 * length // 3, length - 900])]
    m = api.ScoreMatrix.from_text(synth.MATRIX_TEXT, synth.MATRIX_NAME)
    db = api.SubjectDb.from_records(lib)
    enc = [api.encode(q) for q in qs]
    got = []
    for kernels in (0, 1):
        s = api.Searcher(api.SearchParams(**dict(synth.RM_FLAGS, word_size=11, kernels=kernels)), m, db)
        res = s.search(enc)
        got.append((res.counters["so_cells"], res.counters["prelims"], res.tabular("6 score qstart qend sstart send qseq sseq")))
    assert got[0] == got[1]
    assert got[0][2].count("\n") >= 4
