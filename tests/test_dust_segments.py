"""The segmented DUST masker against the sequential pass it replaces (rmb_dust.cuh built for the
host): the words the device lookup tables hold are the words without a masked base."""
import ctypes as C
import subprocess
from pathlib import Path

import numpy as np
import pytest

from rmblast_b200 import api, synth

HERE = Path(__file__).resolve().parent


@pytest.fixture(scope="module")
def dust_host(tmp_path_factory):
    so = tmp_path_factory.mktemp("dust") / "dust_host.so"
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-o", str(so), str(HERE / "dust_host.cpp")],
                   check=True)
    lib = C.CDLL(str(so))
    u8p = C.POINTER(C.c_uint8)
    lib.dust_host.argtypes = [u8p, C.c_uint32, u8p]

    def mask(codes):
        out = codes.copy()
        assert lib.dust_host(codes.ctypes.data_as(u8p), len(codes), out.ctypes.data_as(u8p)) == 0
        return out
    return mask


def stressed(rng, n):
    """Random bases with runs of N, homopolymers (some with an N inside), tandem repeats, single N and
    other codes; some sequences mostly A."""
    g = rng.choice(np.frombuffer(b"ACGT", np.uint8), n, p=[0.85, 0.05, 0.05, 0.05] if rng.random() < 0.25 else None)
    for _ in range(int(rng.integers(0, 8))):
        if n < 12:
            break
        k = min(n, int(rng.integers(10, 160)))
        p = int(rng.integers(0, n - k + 1))
        kind = int(rng.integers(0, 5))
        if kind == 0:
            g[p:p + k] = ord("N")
        elif kind == 1:
            g[p:p + k] = rng.choice(np.frombuffer(b"ACGT", np.uint8))
            if rng.random() < 0.3:
                g[p + int(rng.integers(0, k))] = ord("N")
        elif kind == 2:
            g[p:p + k] = np.resize(synth.random_dna(rng, int(rng.integers(1, 7))), k)
        else:
            g[p] = rng.choice(np.frombuffer(b"NRYMK", np.uint8))
    return g


def with_n_block(rng, n):
    """A sequence with more N than the draws the masker starts with."""
    g = stressed(rng, n)
    g[1000:1000 + 70_000] = ord("N")
    return g


@pytest.mark.gpu
@pytest.mark.parametrize("case", ["edges", "short", "long_units", "many_n"])
def test_segments_mask_what_the_sequential_pass_masks(case, dust_host):
    rng = np.random.default_rng([0xD057, len(case)])
    if case == "edges":  # one window, and around the units of 128 starts with their 62 further steps
        sizes = [*range(7, 10), *range(62, 68), *range(125, 133), *range(187, 195), *range(253, 259), 383, 384, 385, 386]
        seqs = [stressed(rng, n) for n in sizes for _ in range(6)]
    elif case == "short":
        seqs = [stressed(rng, int(rng.integers(20, 2500))) for _ in range(400)]
    elif case == "long_units":  # enough bases for the units of 512 starts
        seqs = [np.concatenate([stressed(rng, 2500) for _ in range(400)]) for _ in range(5)] + [
            stressed(rng, int(rng.integers(500, 2000))) for _ in range(100)]
    else:
        seqs = [with_n_block(rng, 120_000), stressed(rng, 1000), with_n_block(rng, 90_000)]
    db = api.SubjectDb.from_records([("s", synth.random_dna(rng, 200))])
    m = api.ScoreMatrix.from_text(synth.MATRIX_TEXT, synth.MATRIX_NAME)
    s = api.Searcher(api.SearchParams(word_size=7, dust=True), m, db)
    enc = [api.encode(x) for x in seqs]
    # the forward words of each query, as (query, position)
    rows = s.stage(enc, 3)
    first = np.searchsorted(rows[:, 0], np.arange(len(enc) + 1))
    for qi, e in enumerate(enc):
        codes = e[1:-1]
        got = np.zeros(len(codes), bool)
        pos = rows[first[qi]:first[qi + 1], 2]
        got[pos[pos < len(codes)]] = True
        width = 6 if 2 * len(codes) < 250 else 7  # the lookup width of word size 7
        ok = np.convolve(dust_host(codes) < 4, np.ones(width, int), "valid") == width
        want = np.zeros(len(codes), bool)
        want[:len(ok)] = ok
        assert np.array_equal(got, want), (case, qi, len(codes))
