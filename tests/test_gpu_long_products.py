"""Matrix products of long portions (csrc/layered_tc.cu) at the edges of their tiles: token tiles of 32, 64 and 128, weight tiles of 128 rows, stages
of 64, clusters that share a tile's depth; dense, gathered and per-expert products, biased and gated epilogues.

A portion is held against the same tokens one at a time (matrix-vector kernels: the same operands rounded the same way, other sums) and
against the float64 restatement.  Bounds, as root mean squares of a row: two sums of the same bfloat16 products differ by at most
K 2^-24 < 1e-4 of the row, which turns a later operand's last bit (2^-9) here and there; a row whose operands all turned would be off by
2^-9 for each of the six products on its way, 1.2e-2.  Against float64 every operand of every product is rounded, ten roundings of up to 2^-9
on the longest way: 2e-2, of all rows together (a row where the matrix memory's denominator nearly vanishes multiplies its error: 5e-2
in the one-token kernels just the same)."""
import numpy as np
import pytest

from nano_b200 import engine as E, modeldir as md
import fidatar_oracle as F
import kadesun_oracle as K

pytestmark = pytest.mark.gpu


def rel(got, want):
    return float((np.sqrt(((got - want) ** 2).mean(-1)) / np.sqrt((want ** 2).mean(-1))).max())


def model(design, width, ff, vocab):
    if design == "kadesun":
        cfg = md.kadesun_config(vocab, width, [("delta", {"heads": 2, "kv_heads": 1, "dim": 24, "vdim": 40, "conv": 3}, ff),
                                               ("parallel", {"left": {"heads": 4, "kv_heads": 2, "dim": 16, "vdim": 24, "scale": 0.25, "softcap": 20.0, "rot": {"dims": 8, "base": 100.0}},
                                                             "right": {"heads": 2, "kv_heads": 2, "dim": 16, "vdim": 16, "conv": 4}}, ff)])
        return cfg, md.kadesun_random(cfg, 3, decay_rank=8, gate_rank=16), K
    # every expert is chosen by every token, so no close call of the router can tell two right answers apart
    moe = {"kind": "moe", "router": {"experts": 3, "top": 3, "groups": {"count": 1, "keep": 1}, "scale": 0.7}, "expert": {"ff": ff}}
    cfg = md.fidatar_config(vocab, width, [("attention", {"heads": 4, "kv_heads": 2, "dim": 16, "vdim": 24, "scale": 0.25}, moe),
                                           ("mlstm", {"heads": 2, "dim": 24, "vdim": 40, "gate_cap": 8.0}, {"kind": "dense", "ff": ff})], alpha=2.0, scale=2.0)
    return cfg, md.fidatar_random(cfg, 3), F


@pytest.mark.parametrize("design,width,ff,vocab", [("kadesun", 64, 128, 128), ("kadesun", 136, 200, 131), ("kadesun", 520, 1032, 640), ("fidatar", 72, 56, 129), ("fidatar", 256, 264, 300)])
def test_portions_at_tile_edges(tmp_path, design, width, ff, vocab):
    cfg, w, O = model(design, width, ff, vocab)
    eng = E.Engine(md.write_model_dir(str(tmp_path / "m"), cfg, w), 512)
    toks = np.random.default_rng(1).integers(0, vocab, size=257).astype(np.uint32)
    ref = O.forward(cfg, w, toks)
    s = eng.seq_open()
    one = np.concatenate([eng.step(s, toks[i:i + 1], [0]) for i in range(toks.size)])
    eng.seq_close(s)
    for n in (5, 31, 32, 33, 64, 65, 127, 128, 129, 257):
        s = eng.seq_open()
        got = eng.step(s, toks[:n], range(n))
        eng.seq_close(s)
        assert rel(got, one[:n]) < 1.2e-2, n
        assert np.linalg.norm(got - ref[:n]) < 2e-2 * np.linalg.norm(ref[:n]), n
    eng.close()


def test_wide_products(tmp_path):
    """A head of 16392 x 2048, whose tiles would read 32 MB of rows from 32 rows on: on both sides of that line, in copies for tiles of 32 and of 64 tokens.  Bounds as above."""
    cfg = md.kadesun_config(16392, 2048, [("delta", {"heads": 2, "kv_heads": 1, "dim": 24, "vdim": 40, "conv": 3}, None)])
    w = md.kadesun_random(cfg, 3)
    eng = E.Engine(md.write_model_dir(str(tmp_path / "m"), cfg, w), 128)
    toks = np.random.default_rng(1).integers(0, 16392, size=64).astype(np.uint32)
    ref = K.forward(cfg, w, toks)
    s = eng.seq_open()
    one = np.concatenate([eng.step(s, toks[i:i + 1], [0]) for i in range(toks.size)])
    eng.seq_close(s)
    for n in (31, 32, 33, 64):
        s = eng.seq_open()
        got = eng.step(s, toks[:n], range(n))
        eng.seq_close(s)
        assert rel(got, one[:n]) < 1.2e-2, n
        assert np.linalg.norm(got - ref[:n]) < 2e-2 * np.linalg.norm(ref[:n]), n
    eng.close()
