"""How many blocks share a tile's depth (csrc/f32_split.h): a portion's rows count as whole tiles of 64, ragged or not; the largest split whose blocks are at most four
to an SM, with 64 columns of the depth each."""
import os
import subprocess

import pytest

from conftest import ROOT


@pytest.fixture(scope="module")
def probe(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("split") / "probe")
    subprocess.run(["g++", "-O1", "-I" + os.path.join(ROOT, "nano_b200", "csrc"), os.path.join(ROOT, "tests", "f32_split_probe.cpp"), "-o", exe], check=True)
    return lambda *a: int(subprocess.run([exe] + [str(v) for v in a], capture_output=True, text=True, check=True).stdout)


def test_rows_count_as_whole_tiles(probe):
    for cols in (1, 5, 16, 18, 19, 37, 74, 75, 148, 149, 296, 297):
        for rows in (1, 5, 37, 63, 64, 65, 70, 100, 127, 128, 129, 203, 700):
            for groups in (1, 2, 16):
                for K in (4, 64, 128, 1000, 1024, 4096):
                    tiles = cols * -(-rows // 64) * groups
                    fits = [s for s in (1, 2, 4, 8) if s == 1 or tiles * s <= 4 * 148 and K >= s * 64]
                    assert probe(cols, rows, groups, K, 148) == max(fits), (cols, rows, groups, K)


def test_no_product_of_sizes_is_too_large_to_count(probe):
    assert probe(1 << 20, 1 << 20, 64, 4096, 148) == 1
