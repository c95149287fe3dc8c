"""The tensor-core kernels' waits have a limit; what a block does when one runs out is not run (that would take a broken kernel) but read from the source:
a warp that goes on to instructions which all its threads must reach together waits with one verdict for the warp, and warps that
meet at a barrier in a loop leave the loop by the barrier's own answer, not by a word that another warp may set in between."""
import os
import re

import pytest

from conftest import ROOT

# kernel -> where the code of the warps begins that read tensor memory
KERNELS = {"prefill.cu": ("k_prompt_gemm", "} else if (warp >= 2) {"), "attn_tc.cu": ("k_attn_tc", "} else if (warp >= 2) {"), "layered_tc.cu": ("k_gemm_tc", "    if (warp >= 2) {")}


@pytest.mark.parametrize("name", KERNELS)
def test_warps_give_up_together(name):
    kernel, start = KERNELS[name]
    text = re.sub(r"//.*", "", open(os.path.join(ROOT, "nano_b200", "csrc", name)).read())
    body = text[re.search(r"__global__ void __launch_bounds__\([^)]*\) %s\(" % kernel, text).start():]
    body = body[body.index(start):body.index("tc_dealloc")]
    waits = body[:body.rindex("bad_s =")]
    assert "mbar_wait_warp(" in waits and "mbar_wait(" not in waits, "a wait without one verdict for the warp"
    assert "bar.sync" not in waits and "meet()" not in waits, "a barrier whose answer does not say whether to go on"
    assert not re.search(r"bad_s\s*==|!bad_s|\(bad_s\)", waits), "a loop left by a word that other warps set"


def test_warps_that_make_rows_give_up_together():
    """The four warps that finish a tile of k_gemm_tc also bring its rows (tc_rows), where the instance reads them itself: there too a wait has one verdict for the warp, nothing lies between that and the
    return, and the kernel only marks what it is told."""
    text = re.sub(r"//.*", "", open(os.path.join(ROOT, "nano_b200", "csrc", "layered_tc.cu")).read())
    body = text[text.index("bool tc_rows("):]
    body = body[:body.index("\n}\n")]
    waits = re.findall(r"mbar_wait\w*\(", body)
    assert waits and set(waits) == {"mbar_wait_warp("}, "a wait without one verdict for the warp"
    assert len(re.findall(r"!mbar_wait_warp\([^;{}]*\)\) return false;", body)) == len(waits), "a warp goes on after a wait that ran out"
    assert "bar.sync" not in body and "__syncthreads" not in body and "bad_s" not in body
    assert re.search(r"if \(!tc_rows<TN>\([^;{}]*\)\) bad_s = 4;", text)
