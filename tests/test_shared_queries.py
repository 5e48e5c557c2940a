"""One resident query set searched by two contexts at once: its DUST mask and packed copies are made by
whichever search comes first, and both get what each gets alone."""
import threading

import numpy as np
import pytest

from rmblast_b200 import api, synth

FIELDS = "6 score perc_sub qseqid qstart qend sseqid sstart send qseq sseq"


@pytest.mark.gpu
@pytest.mark.parametrize("dust", [False, True])
def test_two_contexts_share_a_fresh_set(dust):
    rng = np.random.default_rng([0x5EA2, dust])
    lib = [synth.random_dna(rng, int(k)) for k in rng.integers(200, 3000, 60)]
    m = api.ScoreMatrix.from_text(synth.MATRIX_TEXT, synth.MATRIX_NAME)
    flags = dict(synth.RM_FLAGS, word_size=11, complexity_adjust=True)
    ctx = [api.Searcher(api.SearchParams(dust=dust, **flags), m,
                        api.SubjectDb.from_records([(f"s{i}", s) for i, s in enumerate(part)]))
           for part in (lib[:30], lib[30:])]
    for rep in range(12):
        qs = []
        for _ in range(20):
            g = synth.plant(rng, synth.random_dna(rng, int(rng.integers(2_000, 40_000))), lib, 0.4, None, (0.02, 0.3), (0.01, 0.05))
            g[500:600] = np.resize(synth.random_dna(rng, 3), 100)
            qs.append(api.encode(g))
        rq = ctx[rep % 2].upload(qs)
        got, gate = [None, None], threading.Barrier(2)

        def search(k):
            gate.wait()
            got[k] = ctx[k].search_resident(rq).tabular(FIELDS)

        threads = [threading.Thread(target=search, args=(k,)) for k in (0, 1)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        rq.free()
        for k in (0, 1):
            want = ctx[k].search(qs).tabular(FIELDS)
            assert want.count("\n") > 20
            assert got[k] == want
