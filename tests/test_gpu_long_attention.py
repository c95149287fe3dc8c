"""Attention of long portions on the tensor cores (csrc/attn_tc.cu) at the edges of its tiles: tiles of 128 keys and of 128 (token, head) rows, head sizes
around 64 and 128, blocks of positions that start inside a tile, a context before the portion, sharp scores.

The portion is held against the same tokens one at a time, whose kernels sum in fp32.  Every product's operands are rounded to bfloat16 the same way
on both sides; the attention differs by its own error of about 1e-6, which turns last bits (2^-9) of later operands here and there: under
1.2e-2 of a row's norm through one layer, of which sharp scores (a factor of 6 on the logits of the softmax) may multiply the part before
them."""
import numpy as np
import pytest

from nano_b200 import engine as E, modeldir as md
import famudra_oracle as A
import fidatar_oracle as F
import vumunex_oracle as V

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("heads,kv,dim,vdim,size,scale", [(4, 1, 32, 32, None, 0.2), (8, 8, 64, 64, None, 0.125), (6, 2, 68, 60, 200, 0.12), (4, 2, 128, 128, None, 0.6), (2, 1, 48, 128, 130, 0.15), (4, 4, 4, 4, 128, 0.5)])
def test_portions_against_single_tokens(tmp_path, heads, kv, dim, vdim, size, scale):
    mixer = {"heads": heads, "kv_heads": kv, "dim": dim, "vdim": vdim, "scale": scale, "rot": {"dims": 4, "base": 100.0}}
    if size:
        mixer["mask"] = {"size": size}
    cfg = md.fidatar_config(64, 96, [("attention", mixer, None)], alpha=0.5, scale=2.0, softcap=None)
    w = md.fidatar_random(cfg, 5)
    eng = E.Engine(md.write_model_dir(str(tmp_path / "m"), cfg, w), 1024)
    toks = np.random.default_rng(2).integers(0, 64, size=600).astype(np.uint32)
    ref = F.forward(cfg, w, toks)
    s = eng.seq_open()
    one = np.concatenate([eng.step(s, toks[i:i + 1], [0]) for i in range(toks.size)])
    eng.seq_close(s)
    for cuts in ([600], [127, 129, 128, 130], [128, 256, 1, 215], [40, 300, 260], [513, 64]):
        s, at, out = eng.seq_open(), 0, []
        for n in cuts:
            out.append(eng.step(s, toks[at:at + n], range(len(toks[at:at + n]))))
            at += n
        eng.seq_close(s)
        got = np.concatenate(out)
        d = np.sqrt(((got - one[:at]) ** 2).mean(-1) / (one[:at] ** 2).mean(-1))
        assert d.max() < 1.2e-2, (cuts, int(d.argmax()))
        assert np.linalg.norm(got - ref[:at]) < 2e-2 * np.linalg.norm(ref[:at]), cuts
    eng.close()


@pytest.mark.parametrize("design,heads,dim,vdim,rank,size", [("famudra", 3, 24, 40, 48, None), ("famudra", 2, 128, 128, 256, None), ("famudra", 5, 64, 68, 8, None), ("vumunex", 3, 20, 12, 40, None), ("vumunex", 4, 64, 64, 128, 130),
                                                            ("vumunex", 2, 128, 60, 72, 200)])
def test_latents_multiplied_out(tmp_path, design, heads, dim, vdim, rank, size):
    """Portions that see 128 keys and more against single tokens (absorbed): the query and the weighted latents are rounded to bfloat16 (2^-9 each) on the
    absorbed side only, so the bound of one layer above stands; plain softmax, window, sink and gate."""
    mixer = {"heads": heads, "dim": dim, "vdim": vdim, "kv_rank": rank, "scale": dim ** -0.5}
    if design == "famudra":
        cfg, make, oracle = md.famudra_config(64, 96, [("latent_attention", dict(mixer, q_rank=56), None)]), md.famudra_random, A.forward
    else:
        cfg = md.vumunex_config(64, 96, [("latent_attention", dict(mixer, mask={"size": size}) if size else mixer, None)], streams=2)
        make, oracle = md.vumunex_random, V.forward
    w = make(cfg, 5)
    eng = E.Engine(md.write_model_dir(str(tmp_path / "m"), cfg, w), 1024)
    toks = np.random.default_rng(2).integers(0, 64, size=600).astype(np.uint32)
    ref = oracle(cfg, w, toks)
    s = eng.seq_open()
    one = np.concatenate([eng.step(s, toks[i:i + 1], [0]) for i in range(toks.size)])
    eng.seq_close(s)
    for cuts in ([600], [127, 5, 129, 128, 130], [130, 6, 464]):
        s, at, out = eng.seq_open(), 0, []
        for n in cuts:
            out.append(eng.step(s, toks[at:at + n], range(n)))
            at += n
        eng.seq_close(s)
        got = np.concatenate(out)
        d = np.sqrt(((got - one[:at]) ** 2).mean(-1) / (one[:at] ** 2).mean(-1))
        assert d.max() < 1.2e-2, (cuts, int(d.argmax()))
        assert np.linalg.norm(got - ref[:at]) < 2e-2 * np.linalg.norm(ref[:at]), cuts
    eng.close()


@pytest.mark.parametrize("design", ["famudra", "vumunex"])
def test_negative_scale(tmp_path, design):
    """A folder may state any number: the most negative product is then the largest score, in portions as in single tokens (bound as above)."""
    mixer = {"heads": 3, "dim": 64, "vdim": 40, "kv_rank": 48, "scale": -0.5}
    if design == "famudra":
        cfg, make, oracle = md.famudra_config(64, 96, [("latent_attention", dict(mixer, q_rank=56), None)]), md.famudra_random, A.forward
    else:
        cfg, make, oracle = md.vumunex_config(64, 96, [("latent_attention", mixer, None)], streams=2), md.vumunex_random, V.forward
    w = make(cfg, 5)
    eng = E.Engine(md.write_model_dir(str(tmp_path / "m"), cfg, w), 512)
    toks = np.random.default_rng(2).integers(0, 64, size=300).astype(np.uint32)
    ref = oracle(cfg, w, toks)
    s = eng.seq_open()
    one = np.concatenate([eng.step(s, toks[i:i + 1], [0]) for i in range(toks.size)])
    eng.seq_close(s)
    s = eng.seq_open()
    got = eng.step(s, toks, range(toks.size))
    eng.close()
    assert np.sqrt(((got - one) ** 2).mean(-1) / (one ** 2).mean(-1)).max() < 1.2e-2
    assert np.linalg.norm(got - ref) < 2e-2 * np.linalg.norm(ref)


def test_no_number_spoils_its_page(tmp_path):
    """A token that is no number: of the tokens before it only those are lost that share its page of 32 keys, in portions with fewer than 128 keys in sight (bound as above)."""
    cfg = md.famudra_config(97, 96, [("latent_attention", {"heads": 4, "dim": 64, "vdim": 64, "kv_rank": 64, "q_rank": 56, "scale": 0.125}, None)])
    w = md.famudra_random(cfg, 5)
    toks = np.random.default_rng(2).integers(0, 96, size=100).astype(np.uint32)
    ref = A.forward(cfg, w, toks)
    toks[70], w["embed"][96] = 96, np.inf
    eng = E.Engine(md.write_model_dir(str(tmp_path / "m"), cfg, w), 128)
    got = eng.step(eng.seq_open(), toks, range(toks.size))
    eng.close()
    assert np.linalg.norm(got[:64] - ref[:64]) < 2e-2 * np.linalg.norm(ref[:64])
    assert np.isnan(got[70:]).all()
