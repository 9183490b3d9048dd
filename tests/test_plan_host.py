"""The rules that cut a step up for its grid (gmt_plan.h), on the CPU: tests/host/plan.cpp prints their choices."""
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
                               (8, 8, 70000), (1, 1, 2000000000), (4, 524280, 2), (4, 524281, 2), (1, 2000000000, 1)])
def test_fp64_passes_fit_the_grid_limits(plan, n):
    """The primitive and predictor passes launch a slab's planes and four (two) more in gridDim.y, the flux
    pass the rows of its tiles; a box that this does not fit has no slab and takes the tile march."""
    (S, _), = plan(("slab", *n))
    assert 0 <= S <= n[2]
    if -(-n[1] // PASS_TY) > GRID_YZ:
        assert S == 0
    else:
        assert 1 <= S and S + 4 <= GRID_YZ
