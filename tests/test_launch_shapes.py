"""Launch shapes and index maps that the kernels rely on, checked on the CPU:
tests/launch_shapes/shapes.cu is compiled against the kernels' own constants
and prints them for every grid length the library dispatches."""
import math
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "paes-channelflow_b200", "csrc")
SRC = os.path.join(ROOT, "tests", "launch_shapes", "shapes.cu")
NVCC = "/usr/local/cuda/bin/nvcc"
SIZES = [16, 32, 64, 96, 128, 192, 256, 384, 512]


@pytest.fixture(scope="module")
def shapes(tmp_path_factory):
    exe = os.path.join(str(tmp_path_factory.mktemp("shapes")), "shapes")
    subprocess.check_call([NVCC, "-std=c++17", "--expt-relaxed-constexpr", "-ccbin", "/usr/bin/g++",
                           "-gencode", "arch=compute_100a,code=sm_100a", "-I", CSRC, SRC, "-o", exe])
    rows = {}
    for line in subprocess.run([exe], capture_output=True, text=True, check=True).stdout.splitlines():
        kind, *rest = line.split()
        rows.setdefault(kind, []).append(rest)
    return rows


def tree_sum(threads):
    """block_sum_store's shuffles over a block of `threads` ones: a lane that
    does not exist gives no defined value."""
    total = 0.0
    for w0 in range(0, threads, 32):
        v = [1.0 if w0 + lane < threads else math.nan for lane in range(32)]
        for o in (16, 8, 4, 2, 1):
            v = [v[lane] + v[lane ^ o] for lane in range(32)]
        total += v[0]
    return total


def test_wall_sums_shuffle_between_lanes_that_exist(shapes):
    """The wall rows' sums (wall_rows_block inside k_clip_walls) go through
    shuffles over whole warps; the row transforms alone would take 126 or 120
    threads at six of the nine lengths."""
    rows = {int(n): (int(t), int(b)) for n, t, b in shapes["clip_walls"]}
    assert sorted(rows) == SIZES
    assert [n for n in SIZES if math.isnan(tree_sum(rows[n][0]))] == [16, 64, 96, 192, 256, 384]
    for n, (threads, block) in rows.items():
        assert threads <= block < threads + 32
        assert tree_sum(block) == block


def test_row_elements_have_one_thread(shapes):
    """k_row_fused has no barrier between a level's last forward pass and the
    next level's first pass: each element that the one reads must be written by
    the same thread in the other."""
    plans = {}
    for real, nsx, t, *rest in shapes["row"]:
        cut = rest.index(":")
        plans.setdefault((int(real), int(nsx)), []).append((rest[:cut], rest[cut + 1:]))
    assert sorted(plans) == [(r, n) for r in (4, 8) for n in SIZES]
    for plan, threads in plans.items():
        owner = {}
        for t, (written, _) in enumerate(threads):
            for e in written:
                assert owner.setdefault(e, t) == t, plan
        assert len(owner) == 3 * plan[1] // 2, plan
        for t, (_, read) in enumerate(threads):
            assert all(owner[e] == t for e in read), (plan, t)


def test_prefetch_tiles_of_the_column_plans(shapes):
    """The tiles that k_y_inverse and k_y_forward prefetch are ColPlan's: boxes
    of at most 256 rows and 256 reals that cover a column exactly, every tile at
    a 16-byte boundary.  Row prefetches: multiples of 16 bytes."""
    seen = set()
    for real, ns, nrows, tc, nb, br in (map(int, r) for r in shapes["tile"]):
        seen.add((real, ns, nrows))
        assert nb * br == nrows and br <= 256, (real, ns, nrows)
        assert (tc * 2 * real) % 16 == 0 and 2 * tc <= 256, (real, ns, nrows)
    assert seen == {(r, n, m) for r in (4, 8) for n in SIZES for m in (n, 3 * n // 2)}
    assert len(shapes["rows"]) == 2 * 2 * len(SIZES)
    assert all(int(b) % 16 == 0 for _, _, b in shapes["rows"])
