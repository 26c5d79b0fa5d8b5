"""Launch shapes of the channel step by dimensions and bins (host arithmetic,
compiled with nvcc, no GPU): which tables stand in shared memory."""
import os
import subprocess

import pytest

from chili_b200 import build

HERE = os.path.dirname(os.path.abspath(__file__))
DIMS = (1, 4, 7, 10, 13, 16, 19, 22)


@pytest.fixture(scope="module")
def shapes(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("shapes") / "channel_shapes")
    subprocess.run([build.nvcc(), *build.ARCH, "-std=c++17", "-I" + os.path.join(build.ROOT, "include"),
                    "-I" + build.CSRC, os.path.join(HERE, "cpp", "channel_shapes.cu"), "-o", exe], check=True)
    pairs = [(d, b) for d in DIMS for b in range(2, 4097)]
    out = subprocess.run([exe], input="".join("%d %d\n" % p for p in pairs), capture_output=True, text=True, check=True)
    return {p: tuple(map(int, line.split())) for p, line in zip(pairs, out.stdout.splitlines())}


def test_batched_tasks_keep_their_tables_in_shared_memory(shapes):
    """Every table that the grouped launches staged with two-cell hints and
    edges (up to 48 KB) is staged as cells and widths too, except where these
    leave no room for 32 warps (7 dimensions from 257 bins on, 137 KB)."""
    for (d, b), s in shapes.items():
        hint_tables = 8 * d * (2 * b + 1) + 4 * d * 2 * b + d
        if hint_tables <= 48 * 1024 and d > 1:
            assert s[3] or (d, b >= 257) == (7, True), (d, b)


def test_shapes_fit_a_multiprocessor(shapes):
    for (d, b), s in shapes.items():
        for tables, smem, threads in (s[:3], s[3:]):
            assert smem <= 200 * 1024 and threads in (256, 512, 1024) and (threads < 1024 or 10 < d <= 16), (d, b)
            assert tables or smem < 1024
        assert not s[3] or (228 * 1024 // (s[4] + 1024)) * s[5] >= 1024, (d, b)  # 32 warps beside the tables
