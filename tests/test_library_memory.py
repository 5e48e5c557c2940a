"""The packed DP's copy of the library (three bytes a base) is made only for parameters that use it."""
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
