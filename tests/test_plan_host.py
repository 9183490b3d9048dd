"""Host code of the library without a GPU: the rules that cut a step up for its grid (gmt_plan.h; tests/host/plan.cpp
prints their choices), and the turns at shared scratch (gmt_turn.h)."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
GRID_YZ = 65535                 # largest gridDim.y and gridDim.z of a launch
PASS_TY = 8                     # rows per block of the FP64 flux pass


@pytest.fixture(scope="module")
def plan(tmp_path_factory):
    cxx = shutil.which("g++") or shutil.which("c++")
    if not cxx:
        pytest.skip("no C++ compiler")
    exe = str(tmp_path_factory.mktemp("plan") / "plan")
    subprocess.run([cxx, "-std=c++17", "-O1", "-Wall", "-Werror", "-o", exe, os.path.join(HERE, "host", "plan.cpp")], check=True)

    def ask(*queries):
        text = "\n".join(" ".join(str(x) for x in q) for q in queries)
        out = subprocess.run([exe], input=text, check=True, capture_output=True, text=True).stdout
        rows = [[int(x) for x in line.split()] for line in out.splitlines()]
        assert len(rows) == len(queries)
        return rows
    return ask


# narrow boxes of many planes and of many rows among ordinary ones, all within gmt_create's 4e9 cells
@pytest.mark.parametrize("n", [(1, 1, 1), (16, 16, 16), (192, 192, 192), (512, 512, 512), (8, 8, 65531), (8, 8, 65532),
                               (8, 8, 70000), (1, 1, 2000000000), (1, 524280, 2), (1, 524281, 2), (1, 2000000000, 1)])
def test_fp64_passes_fit_the_grid_limits(plan, n):
    """The primitive and predictor passes launch a slab's planes and four (two) more in gridDim.y, the flux
    pass the rows of its tiles; a box that this does not fit has no slab and takes the tile march."""
    (S, _), = plan(("slab", *n, 1))
    assert 0 <= S <= n[2]
    if -(-n[1] // PASS_TY) > GRID_YZ:
        assert S == 0
    else:
        assert 1 <= S and S + 4 <= GRID_YZ


# cross sections around the one whose four planes just fit, thin and thick; the boxes of an ensemble
@pytest.mark.parametrize("n", [(192, 192, 192), (1024, 1024, 3), (1024, 1024, 64), (1029, 1029, 64), (1030, 1030, 64),
                               (1536, 1536, 3), (1536, 1536, 128), (2048, 2048, 256), (1024, 1024, 9), (512, 512, 512), (528, 528, 528)])
@pytest.mark.parametrize("lanes", [1, 3, 4])
def test_fp64_scratch_stays_within_its_budget(plan, n, lanes):
    """The passes' scratch is at most 1 GB for a context and for all lanes of an ensemble together; slabs are cut
    down to three or four planes (or the box's, if it has fewer), and a box that still exceeds it has none."""
    (S, size), = plan(("slab", *n, lanes))
    budget = (1 << 30) // lanes
    if S == 0:   # 9 planes of primitives and of predictors in 8 bytes, 4 and 2 more than the slab; 1-byte flags
        k = min(4, n[2])
        assert n[0] * n[1] * (72 * (2 * k + 6) + k + 2) > budget
    else:
        assert S >= min(3, n[2]) and size <= budget


def test_scratch_is_handed_on_however_a_holder_leaves(tmp_path):
    """ScratchTurn (gmt_turn.h) over stand-ins of the runtime calls (tests/host/turn.cpp): a holder that leaves
    by an error exit after launching has its work marked like any other; one that could not wait for the last
    holder neither launches nor marks; work that cannot be marked is waited for."""
    cuda = "/usr/local/cuda/include"
    cxx = shutil.which("g++") or shutil.which("c++")
    if not cxx or not os.path.exists(os.path.join(cuda, "cuda_runtime_api.h")):
        pytest.skip("no C++ compiler or CUDA headers")
    exe = str(tmp_path / "turn")
    subprocess.run([cxx, "-std=c++17", "-O1", "-Wall", "-Werror", "-pthread", "-I", cuda, "-o", exe,
                    os.path.join(HERE, "host", "turn.cpp")], check=True)
    out = subprocess.run([exe], check=True, capture_output=True, text=True, timeout=60).stdout
    got = [s.split("\n")[:-1] for s in out.split("end\n")[:-1]]
    assert got[0] == ["wait 1", "launch 1", "record 1", "status 0", "free 1"]
    assert got[1] == ["wait 1", "launch 1", "record 1", "status 1", "free 1"]
    assert got[2] == ["wait 1", "status 1", "free 1"]
    assert got[3] == ["wait 1", "launch 1", "record 1", "synchronise 1", "status 1", "free 1"]
    assert got[4] == ["wait 1", "launch 1", "record 1", "wait 2", "launch 2", "record 2"]
