"""The parts of a prompt product's depth (csrc/prompt_split.h) for every depth and group size that a Q80 or F32 file may have: in order, without gaps,
and n / group size groups in all -- also where the last blocks of a cluster get no stage of a depth that is no multiple of 128."""
import os
import subprocess

from conftest import ROOT


def test_parts_cover_every_depth(tmp_path):
    exe = str(tmp_path / "probe")
    subprocess.run(["g++", "-O1", "-I" + os.path.join(ROOT, "nano_b200", "csrc"), os.path.join(ROOT, "tests", "prompt_split_probe.cpp"), "-o", exe], check=True)
    r = subprocess.run([exe, "32768"], capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout
