"""How many query heads an attention item of the streaming kernel takes (csrc/stream_groups.h): the fewest whose items, a key/value head's keys dealt out over the SMs, hold at most 20480 coordinates
of keys; all of them where none do, and in Q4K files."""
import os
import subprocess

import pytest

from conftest import ROOT


@pytest.fixture(scope="module")
def probe(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("groups") / "probe")
    subprocess.run(["g++", "-O1", "-I" + os.path.join(ROOT, "nano_b200", "csrc"), os.path.join(ROOT, "tests", "stream_groups_probe.cpp"), "-o", exe], check=True)
    return lambda *a: tuple(int(v) for v in subprocess.run([exe] + [str(int(v)) for v in a], capture_output=True, text=True, check=True).stdout.split())


def test_items_hold_what_the_ring_holds(probe):
    for kv in (1, 3, 8, 16, 74, 75, 148):
        for mul in (1, 2, 4):
            for hd in (12, 48, 64, 128):
                for keys in (1, 31, 320, 321, 1440, 1441, 2880, 40960):
                    splits = {h: min(64, max(1, 148 // (kv * mul // h))) for h in (1, 2, 4) if h <= mul}
                    fits = [h for h in splits if kv * mul // h <= 148 and keys * hd <= 20480 * splits[h]]
                    want = min(fits) if fits else mul
                    assert probe(kv, mul, hd, False, keys, 148) == (want, splits[want]), (kv, mul, hd, keys)
                    assert probe(kv, mul, hd, True, keys, 148)[0] == mul
