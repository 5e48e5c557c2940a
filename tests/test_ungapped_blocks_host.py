"""The kernels' ungapped walk (UngBlocks of rmb_ungapped.cuh: eight bases a step from aligned words), built for
the host by tests/ungapped_blocks_host.cu, against the oracle's extension (search/ungapped.rs:38-121)."""
import re
import shutil
import subprocess
from pathlib import Path

import pytest

import oracle_ref as O

ROOT = Path(__file__).resolve().parent.parent
pytestmark = pytest.mark.skipif(shutil.which("nvcc") is None and not Path("/usr/local/cuda/bin/nvcc").exists(),
                                reason="nvcc not found")


@pytest.fixture(scope="module")
def harness(tmp_path_factory):
    O.build_oracle()
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    out = tmp_path_factory.mktemp("ungapped_blocks_host") / "ungapped_blocks_host"
    lib = ROOT / "oracle" / "build"
    subprocess.run([nvcc, "-std=c++17", "-O2", "-o", str(out), str(ROOT / "tests" / "ungapped_blocks_host.cu"),
                    "-L", str(lib), "-lrmb_oracle", "-Xlinker", "-rpath", "-Xlinker", str(lib)], check=True)
    return out


@pytest.mark.parametrize("seed,xdrop", [(1, 0), (2, 20), (3, 100), (4, 400), (5, 2**31 - 1)])
def test_walk_matches_oracle(harness, seed, xdrop):
    r = subprocess.run([str(harness), "20000", str(seed), str(xdrop), str(O.GOLDEN / "comparison.matrix")],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    v = dict((k, int(x)) for k, x in re.findall(r"(\w+) (\d+)", r.stdout))
    assert v["bad"] == 0 and v["hits"] == 20000 and v["steps"] > 20000
