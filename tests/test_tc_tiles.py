"""Which products of a portion read their rows themselves (csrc/tc_tiles.h): groups of one tile of 32 or 64 tokens, while all tiles of 128 columns together read at most 32 MB; the rest, and every
group of more than 64, works on a rounded copy.  Several tokens' tiles of one group always have 128, so the split of a depth, and with it the order of a sum, does not
follow from where rows are read."""
import os
import subprocess

from conftest import ROOT


def test_who_reads_rows(tmp_path):
    exe = str(tmp_path / "probe")
    subprocess.run(["g++", "-O1", "-I" + os.path.join(ROOT, "nano_b200", "csrc"), os.path.join(ROOT, "tests", "tc_tiles_probe.cpp"), "-o", exe], check=True)
    sizes = [(n, g, e, k) for n in (1, 128, 129, 2048, 8192, 8193, 12288, 16384, 16385, 152064) for g in (1, 3, 16, 64) for e in (1, 5, 31, 32, 33, 63, 64, 65, 128, 129, 384, 385, 4096)
             for k in (8, 520, 1024, 2048, 2056, 8192)]
    out = subprocess.run([exe], input="\n".join(" ".join(map(str, s)) for s in sizes), capture_output=True, text=True, check=True).stdout.split()
    got = list(zip(map(int, out[::2]), map(int, out[1::2])))
    assert len(got) == len(sizes)
    for (n, g, e, k), (tokens, reads) in zip(sizes, got):
        assert tokens == (32 if e <= 32 else 64 if e <= 64 else 128), (n, g, e, k)
        assert reads == (e <= 64 and -(-n // 128) * g * e * k * 4 <= 32 << 20), (n, g, e, k)
