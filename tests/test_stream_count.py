"""What the host counts of the streaming kernel's launches (csrc/stream_count.h) stays what the device has counted when launches are refused: a launch that
started from arrivals which never came would wait for them in vain."""
import os
import re
import subprocess

from conftest import ROOT

CSRC = os.path.join(ROOT, "nano_b200", "csrc")


def test_refused_launches_count_for_nothing(tmp_path):
    exe = str(tmp_path / "probe")
    subprocess.run(["g++", "-O1", "-I" + CSRC, os.path.join(ROOT, "tests", "stream_count_probe.cpp"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout


def test_every_launch_of_the_kernel_is_counted_there():
    text = re.sub(r"//.*", "", open(os.path.join(CSRC, "engine.cu")).read())
    assert len(re.findall(r"cudaLaunchCooperativeKernel\(e->st_kern", text)) == 1 and len(re.findall(r"g\.(?:epoch_base|bar_base) =", text)) == 2
    body = text[text.index("e->st_count.run("):]
    assert body.index("g.epoch_base =") < body.index("cudaLaunchCooperativeKernel(e->st_kern") < body.index("});")
