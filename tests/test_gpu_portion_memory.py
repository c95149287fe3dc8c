"""The workspaces of long portions and prompts are optional: they take at most an eighth of what is free after the engine itself, and a context that they
have no room for runs on the kernels that need none.  Memory is made short by an allocation of the test's own.  Bounds of the logits as in
test_gpu_long_attention.py and test_gpu_prompts.py."""
import numpy as np
import pytest
import torch

from nano_b200 import engine as E, modeldir as md, modelfile as mf

pytestmark = pytest.mark.gpu
MB = 1 << 20


def free():
    return torch.cuda.mem_get_info()[0]


class Short:
    """All but `leave` bytes of the device's memory are taken."""

    def __init__(self, leave):
        torch.cuda.empty_cache()
        self.held = torch.empty(free() - leave, dtype=torch.uint8, device="cuda")

    def __enter__(self):
        return self

    def __exit__(self, *_):
        self.held = None
        torch.cuda.empty_cache()


def opened(path, room):
    before = free()
    eng = E.Engine(path, room)
    return eng, before - free(), E.lib().nb200_last_error().decode()


def rel(a, b):
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


@pytest.mark.parametrize("leave", [512 * MB, 100 * MB])
def test_folder(tmp_path, leave):
    mixer = {"heads": 16, "dim": 64, "vdim": 64, "kv_rank": 64, "q_rank": 64, "scale": 0.125}
    cfg = md.famudra_config(64, 128, [("latent_attention", mixer, None)])
    path = md.write_model_dir(str(tmp_path / "m"), cfg, md.famudra_random(cfg, 5))
    toks = np.random.default_rng(2).integers(0, 64, size=4000).astype(np.uint32)

    def logits(eng):
        s = eng.seq_open()
        out = np.concatenate([eng.step(s, toks[:600], [0, 300, 599]), eng.step(s, toks[600:], [10, 3399])])
        eng.seq_close(s)
        return out

    eng = E.Engine(path, 8192)          # kernels are loaded for good
    logits(eng)
    eng.close()
    eng, ample, said = opened(path, 32768)
    want = logits(eng)
    eng.close()
    assert said == "" and ample > 500 * MB
    with Short(leave):
        eng, used, said = opened(path, 32768)
        got = logits(eng)
        eng.close()
    assert used < 64 * MB + leave / 8 and "need no workspace" in said, (used, said)
    assert (np.linalg.norm(got - want, axis=1) / np.linalg.norm(want, axis=1)).max() < 1.2e-2


@pytest.mark.parametrize("quant", [mf.QUANT_Q80, mf.QUANT_F32])
def test_file(quant):
    spec = mf.ModelSpec("portion-memory", mf.ARCH_QWEN3, 32768, 512, 2, 256, 8, 8, 512, 128)
    path = mf.cached_model(spec, quant, 64)
    ids = np.zeros(2402, np.uint32)
    ids[:2400] = mf.teacher_tokens(2400, 512)
    eng = E.Engine(path, 512)          # kernels are loaded for good
    eng.forward_nolog(0, 0)
    eng.decode_greedy(ids[:202].copy(), 200, 202)
    eng.close()
    eng, ample, said = opened(path, 32768)
    assert said == ""
    want = []
    for n in (200, 2400):
        for p in range(n):
            eng.forward_nolog(int(ids[p]), p)
        want.append(eng.logits())
    eng.close()
    with Short(ample):          # room for all of it but not within an eighth
        eng, used, said = opened(path, 32768)
        got = []
        for n in (200, 2400):
            eng.decode_greedy(ids.copy(), n, n + 1)
            got.append(eng.logits())
        eng.close()
    assert used < ample - 150 * MB, (used, ample, said)
    for g, w in zip(got, want):
        assert rel(g, w) < (1e-5 if quant == mf.QUANT_F32 else 4e-2)
