"""Host code of the library without a GPU: the rules that cut a step up for its grid (gmt_plan.h; tests/host/plan.cpp
prints their choices), the turns at shared scratch (gmt_turn.h), and what is kept for later steps (gmt_recent.h)."""
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


@pytest.mark.parametrize("units,mean,lanes", [(1, 192 ** 3, 1), (2, 256 ** 3, 2), (3, 128 ** 3, 3), (4, 112 ** 3, 4), (64, 32 ** 3, 4),
                                              (4, 128 ** 3, 2), (64, 192 ** 3, 2), (64, (60 * 32 ** 3 + 4 * 128 ** 3) // 64, 4)])
def test_fp64_lanes_keep_a_mean_box_whole_where_two_of_them_can(plan, units, mean, lanes):
    (got,), = plan(("lanes", units, mean))
    assert got == lanes


# dtype, boxes by size, us a step of the ensemble with a launch for each box and with those of a size together
BATCHES = [
    ("f32", {16: 64}, 213, 79), ("f32", {16: 512}, 1297, 413), ("f32", {32: 64}, 342, 280), ("f32", {32: 256}, 1231, 888),
    ("f32", {16: 100, 128: 1}, 514, 328), ("f32", {32: 32, 48: 4}, 256, 231), ("f32", {32: 5, 48: 1}, 79, 72),
    ("f32", {32: 6, 48: 3, 64: 1}, 132, 141), ("f32", {32: 14, 48: 8, 64: 12}, 506, 550), ("f32", {32: 8, 64: 8}, 254, 279),
    ("f32", {32: 13, 48: 13, 64: 12, 96: 13, 128: 13}, 4025, 4093), ("f32", {48: 64}, 798, 794),
    ("f64", {16: 4}, 99, 149), ("f64", {16: 16}, 372, 152), ("f64", {16: 256}, 6075, 1017), ("f64", {16: 100, 128: 1}, 5731, 2191),
    ("f64", {16: 3, 256: 1}, 8740, 9217),
]


@pytest.mark.parametrize("dtype,boxes,alone,together", BATCHES)
def test_small_boxes_share_launches_where_that_is_faster(plan, dtype, boxes, alone, together):
    """Boxes of 16^3 (and in FP32 of 32^3) share launches where the ensemble was measured faster by more than 3 % for
    it, and do not where it was slower by as much as 1 %."""
    mean = sum(c * n ** 3 for n, c in boxes.items()) // sum(boxes.values())
    esize = 8 if dtype == "f64" else 4
    got = {n: c for n, (c,) in zip(boxes, plan(*[("batch", esize, n, c, mean) for n, c in boxes.items()]))}
    assert all(1 <= got[n] <= min(c, 64) for n, c in boxes.items())
    assert all(c == 1 for n, c in got.items() if n > (16 if dtype == "f64" else 32))
    shares = max(got.values()) > 1
    if together < 0.97 * alone:
        assert shares
    if together > 1.01 * alone:
        assert not shares


# us a step of a tile march: with the rule that asked for eight rounds of blocks and no more (the kernels of
# that time), and by planes per block.  Tiles of which several blocks share an SM:
CHUNK_TIMES = [
    ("unsplit mc", (64, 64, 64), "f32", (8, 8), 82, {4: 86, 6: 71, 8: 76, 12: 97, 16: 114, 24: 163, 32: 204, 64: 351}),
    ("unsplit mc", (64, 64, 64), "f32", (16, 8), 67, {4: 77, 6: 59, 8: 62, 12: 87, 16: 106, 24: 137, 32: 178, 64: 329}),
    ("unsplit ppm", (64, 64, 64), "f32", (32, 4), 104, {4: 131, 6: 95, 8: 104, 12: 142, 16: 175, 24: 243, 32: 315, 64: 603}),
    ("unsplit mc", (128, 128, 128), "f32", (16, 8), 380, {4: 405, 6: 363, 8: 342, 12: 331, 16: 353, 24: 349, 32: 437, 64: 410, 128: 729}),
    ("unsplit ppm", (128, 128, 128), "f32", (32, 8), 547, {4: 530, 6: 511, 8: 517, 12: 540, 16: 513, 24: 668, 32: 514, 64: 736, 128: 1419}),
    ("unsplit mc", (128, 128, 128), "f32", (16, 16), 308, {4: 241, 6: 228, 8: 228, 12: 228, 16: 222, 24: 267, 32: 223, 64: 337, 128: 599}),
    ("march1d mc", (128, 128, 128), "f32", (16, 8), 308, {4: 332, 6: 293, 8: 279, 12: 270, 16: 287, 24: 283, 32: 354, 64: 340, 128: 611}),
    ("ct mc", (128, 128, 128), "f32", (16, 8), 353, {4: 357, 6: 324, 8: 308, 12: 306, 16: 326, 24: 326, 32: 403, 64: 376, 128: 656}),
    ("unsplit mc", (128, 64, 96), "f32", (32, 4), 225, {4: 164, 6: 162, 8: 149, 12: 186, 16: 142, 24: 159, 32: 209, 48: 294, 64: 388}),
    ("unsplit mc", (256, 256, 256), "f32", (16, 8), 2249, {4: 3133, 6: 2816, 8: 2647, 12: 2462, 16: 2325, 24: 2192, 32: 2194, 64: 2166, 128: 2509}),
    ("unsplit mc", (64, 64, 64), "f64", (8, 8), 506, {4: 401, 6: 385, 8: 499, 12: 380, 16: 491, 24: 726, 32: 949, 64: 1806}),
    ("unsplit mc", (128, 64, 96), "f64", (8, 8), 1004, {4: 952, 6: 975, 8: 1019, 12: 1114, 16: 996, 24: 1425, 32: 990, 64: 1930, 96: 2792}),
    ("ct mc", (128, 128, 128), "f64", (8, 8), 2999, {4: 3262, 6: 3140, 8: 3133, 12: 3115, 16: 3052, 24: 3167, 32: 3382, 64: 3403, 128: 3380}),
    # one block fills an SM
    ("unsplit mc", (128, 128, 128), "f64", (16, 16), 1725, {4: 1746, 6: 1718, 8: 1654, 12: 1711, 16: 1817, 24: 1981, 32: 1801, 64: 1779, 128: 3363}),
    ("unsplit ppm", (128, 128, 128), "f64", (32, 8), 2985, {4: 3107, 6: 3046, 8: 2964, 12: 3065, 16: 3274, 24: 3554, 32: 3245, 64: 3166, 128: 6051}),
    ("unsplit ppm", (128, 128, 128), "f64", (16, 8), 6062, {4: 6458, 6: 6243, 8: 6128, 12: 6140, 16: 5961, 24: 6275, 32: 6682, 64: 6661, 128: 6573}),
    ("unsplit ppm", (128, 64, 96), "f64", (16, 16), 1240, {4: 1244, 6: 1219, 8: 1200, 11: 1091, 12: 1181, 16: 1531, 24: 1142, 32: 1471, 64: 2897}),
    ("unsplit mc", (128, 64, 96), "f64", (16, 8), 1358, {4: 1437, 6: 1337, 8: 1441, 11: 1326, 12: 1446, 16: 1442, 24: 1429, 32: 1846, 48: 1398, 64: 1831}),
    ("march1d mc", (128, 128, 128), "f64", (16, 8), 1451, {4: 1656, 6: 1536, 8: 1485, 12: 1439, 16: 1426, 24: 1405, 32: 1485, 64: 1479, 128: 1533}),
    ("ct mc", (128, 64, 96), "f64", (16, 8), 1139, {4: 1202, 6: 1144, 8: 1229, 11: 1130, 12: 1231, 16: 1239, 24: 1230, 32: 1573, 48: 1216, 64: 1581}),
    ("ct mc", (64, 64, 64), "f64", (16, 8), 420, {4: 439, 6: 465, 8: 425, 12: 568, 16: 408, 24: 576, 32: 740, 64: 1491}),
    ("march1d ppm", (128, 128, 128), "f64", (16, 16), 2569, {4: 2683, 8: 2554, 10: 2622, 12: 2638, 16: 2802, 20: 2637, 24: 3017, 32: 2796, 40: 3375, 48: 3292, 64: 2734, 80: 3340}),
    ("march1d mc", (96, 96, 96), "f64", (16, 16), 366, {4: 380, 8: 339, 10: 399, 12: 327, 16: 413, 20: 454, 24: 316, 32: 408, 40: 502}),
    ("march1d ppm", (160, 160, 160), "f64", (16, 16), 4970, {4: 5187, 8: 5069, 10: 4957, 12: 4883, 16: 4969, 20: 5234, 24: 5015, 32: 5542, 40: 5215, 48: 5898, 64: 5511, 80: 6854, 128: 5514}),
    ("ct mc", (128, 128, 128), "f64", (16, 8), 3039, {4: 3056, 8: 2924, 10: 2956, 12: 2909, 16: 2857, 20: 2944, 24: 2989, 32: 3201, 40: 3007, 48: 3175, 64: 3192, 80: 3184, 128: 3146}),
    ("ct ppm", (128, 128, 128), "f64", (16, 8), 5595, {4: 5657, 8: 5425, 10: 5498, 12: 5393, 16: 5306, 20: 5472, 24: 5547, 32: 5924, 40: 5580, 48: 5875, 64: 5922, 80: 5909, 128: 5800}),
    ("ct mc", (112, 112, 112), "f64", (16, 8), 2043, {4: 2082, 8: 2072, 10: 2049, 12: 1956, 16: 2039, 20: 2012, 24: 2049, 32: 2023, 38: 1903, 40: 1986, 48: 2358, 64: 2398, 80: 2015}),
    ("ct mc", (144, 144, 144), "f64", (16, 8), 4141, {4: 4311, 8: 4154, 10: 4075, 12: 4145, 16: 4090, 20: 4053, 24: 4229, 32: 4044, 40: 4210, 48: 4713, 64: 4628, 80: 5054, 128: 5989}),
]


@pytest.mark.parametrize("what,n,dtype,tile,before,times", CHUNK_TIMES)
def test_chunks_are_no_slower_than_eight_rounds_of_blocks(plan, what, n, dtype, tile, before, times):
    """The planes per block that the rule takes were measured no slower than what it replaced (2 %: two runs)."""
    cols = -(-n[0] // tile[0]) * -(-n[1] // tile[1])
    (lz,), = plan(("chunk", cols, n[2], 8 if dtype == "f64" else 4, tile[0] * tile[1]))
    assert lz in times, lz
    assert times[lz] <= 1.02 * before


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
    assert got[5] == ["wait 1", "record 1", "wait 2", "launch 2", "record 2"]


def test_tensor_maps_kept_for_later_steps_are_whole(tmp_path):
    """What a context keeps of its last input states (gmt_recent.h), under threads that step on more states than
    it holds: a map that another thread was writing would be handed to the TMA unit."""
    cxx = shutil.which("g++") or shutil.which("c++")
    if not cxx:
        pytest.skip("no C++ compiler")
    exe = str(tmp_path / "recent")
    subprocess.run([cxx, "-std=c++17", "-O2", "-Wall", "-Werror", "-pthread", "-o", exe, os.path.join(HERE, "host", "recent.cpp")],
                   check=True)
    found, torn, oldest, rest = subprocess.run([exe], check=True, capture_output=True, text=True, timeout=120).stdout.split()
    assert int(found) > 0 and int(torn) == 0
    assert oldest == "0" and rest == "1111"
