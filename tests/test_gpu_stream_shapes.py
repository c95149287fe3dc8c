"""The streaming decode kernel over the shapes its instances and row blocks are chosen by, against the oracle: query heads per kv head x head sizes
(lanes of a cache row), attention items of one pass, of several segments and merged over several CTAs, rows shorter and longer than a warp's step."""
import numpy as np
import pytest

from nano_b200 import engine as E, modelfile as mf
from oracle import bindings as ob

pytestmark = pytest.mark.gpu

#          arch           heads kv  head  width  hidden
SHAPES = [(mf.ARCH_NANO, 2, 2, 12, 24, 20), (mf.ARCH_NANO, 4, 4, 48, 192, 36), (mf.ARCH_NANO, 4, 2, 100, 400, 64), (mf.ARCH_QWEN3, 3, 3, 128, 96, 260),
          (mf.ARCH_QWEN3, 4, 2, 64, 1028, 300), (mf.ARCH_QWEN3, 4, 2, 128, 64, 516), (mf.ARCH_QWEN3, 4, 1, 32, 128, 128), (mf.ARCH_QWEN3, 8, 2, 128, 64, 2052)]
#        rows of an attention item, ring stage in KB: default; 8 rows (many items); several segments per item
PLANS = [(0, 16), (8, 16), (512, 5)]


def run(spec, quant, gs, chunk, stage, monkeypatch, n):
    monkeypatch.setenv("NB200_STREAM", "1")
    monkeypatch.setenv("NB200_STAGE_KB", str(stage))
    if chunk:
        monkeypatch.setenv("NB200_ATTN_CHUNK", str(chunk))
    path = mf.cached_model(spec, quant, gs)
    eng = E.Engine(path, n)
    assert eng.path.startswith("streaming"), eng.path
    o = ob.NanoOracle(path, n)
    toks = mf.teacher_tokens(n, spec.vocab)
    a, b = np.zeros((2, n, spec.vocab))
    for pos in range(n):
        a[pos], b[pos] = eng.forward(toks[pos], pos), o.forward(toks[pos], pos)
    eng.close()
    o.close()
    return a, b


@pytest.mark.parametrize("chunk,stage", PLANS)
@pytest.mark.parametrize("arch,H,KV,hd,E_,F", SHAPES)
def test_f32_shapes(arch, H, KV, hd, E_, F, chunk, stage, monkeypatch):
    spec = mf.ModelSpec("shape-%d-%d-%d-%d-%d-%d" % (arch, H, KV, hd, E_, F), arch, 128, 97, 2, E_, H, KV, F, hd)
    if chunk == 512 and (stage * 1024 // (8 * hd)) * 8 >= 75:
        pytest.skip("one segment holds the whole context of so small a head")
    a, b = run(spec, mf.QUANT_F32, 128, chunk, stage, monkeypatch, 75)
    # both sides hold 24 bits in every sum: rows of up to 2052 products and 75 weighted rows, through two layers, differ by their order
    # only, about sqrt(2052) * 2^-24 = 3e-6 of a row's size a layer at most
    assert np.linalg.norm(a - b) <= 1e-5 * np.linalg.norm(b)


# contexts at the edge of the rule for the query heads of an attention item (640 keys of 32 where every query head's item has all keys): the tokens on both sides of it against the oracle,
# and a device loop over the edge gives the bits of one call per token
@pytest.mark.parametrize("H,KV,hd,edge", [(80, 40, 32, 640), (80, 20, 32, 640)])
def test_heads_of_an_item(H, KV, hd, edge, monkeypatch):
    monkeypatch.setenv("NB200_STREAM", "1")
    n = edge + 6
    spec = mf.ModelSpec("heads-%d-%d-%d" % (H, KV, hd), mf.ARCH_QWEN3, 1024, 97, 1, 64, H, KV, 64, hd)
    path = mf.cached_model(spec, mf.QUANT_F32, 128)
    eng, o = E.Engine(path, n + 2), ob.NanoOracle(path, n + 2)
    assert eng.path.startswith("streaming"), eng.path
    ids = np.zeros(n + 2, np.uint32)
    ids[:4] = 5, 7, 9, 11
    eng.decode_greedy(ids, 4, n + 1)
    loop = eng.logits()
    for pos in range(n):
        a, b = eng.forward(int(ids[pos]), pos), o.forward(int(ids[pos]), pos)
        if pos >= edge - 4:
            assert np.linalg.norm(a - b) <= 1e-5 * np.linalg.norm(b), pos          # as above
    assert np.array_equal(a, loop)
    eng.close()
    o.close()


# widths of one quantisation group, of an odd number of them, of more than one 1024-byte step of a warp, and of more than one turn of the prologue's warps
@pytest.mark.parametrize("E_,F,gs", [(64, 64, 64), (192, 320, 64), (640, 1152, 128), (128, 4224, 128), (3968, 128, 128)])
def test_q80_rows(E_, F, gs, monkeypatch):
    spec = mf.ModelSpec("rows-%d-%d-%d" % (E_, F, gs), mf.ARCH_QWEN3, 128, 131, 1, E_, 4, 2, F, 64 if E_ != 3968 else 128)
    a, b = run(spec, mf.QUANT_Q80, gs, 0, 16, monkeypatch, 20)
    # sums in another order turn an activation code here and there, by one of 127 steps of its group: 2^-8 of a row's size at most, where not so it is 1e-6
    assert np.linalg.norm(a - b) <= 4e-3 * np.linalg.norm(b)
    assert np.median(np.linalg.norm(a - b, axis=1) / np.linalg.norm(b, axis=1)) <= 2e-3


def test_logits_are_those_of_the_last_step(monkeypatch):
    """forward leaves its logits in pinned host memory; whatever runs afterwards must not be answered from there."""
    monkeypatch.setenv("NB200_STREAM", "1")
    spec = mf.PRESETS["toy-qwen3"]
    eng = E.Engine(mf.cached_model(spec, mf.QUANT_Q80, 64), 64)

    def device():
        return eng.read(E.F_LOGITS, spec.vocab)
    a = eng.forward(5, 0)
    assert np.array_equal(a, device())
    b = eng.forward(7, 1)
    assert np.array_equal(b, device()) and not np.array_equal(a, b)
    eng.next_greedy(np.array([5, 7, 9, 0], np.uint32), 2, 0)
    c = eng.logits()
    assert np.array_equal(c, device()) and not np.array_equal(b, c)
    assert np.array_equal(eng.forward(9, 2), c)
    ids = np.zeros(40, np.uint32)
    ids[:3] = [5, 7, 9]
    eng.decode_greedy(ids, 3, 20)
    d = eng.logits()
    assert np.array_equal(d, device()) and not np.array_equal(c, d)
    assert eng.next_greedy(ids, 19, 0) == int(np.argmax(eng.logits()))
    eng.close()


@pytest.mark.parametrize("quant,gs", [(mf.QUANT_F32, 128), (mf.QUANT_Q80, 64), (mf.QUANT_Q80, 128), (mf.QUANT_Q4K, 128)])
@pytest.mark.parametrize("arch", [mf.ARCH_NANO, mf.ARCH_QWEN3])
def test_rows_whose_squares_overflow(arch, quant, gs, monkeypatch, tmp_path):
    """The sum of squares of every third token's row is infinite in 32 bits and one over its root zero: such a row norms to zeros, as in the oracle, and gives zeros
    for logits and for its keys and values; the tokens between have theirs within the bounds above (Q4K: as finite numbers)."""
    monkeypatch.setenv("NB200_STREAM", "1")
    spec = mf.ModelSpec("overflow-%d-%d-%d" % (arch, quant, gs), arch, 128, 96, 2, 256, 4, 2, 256, 64)
    rng = np.random.default_rng(11)
    L, W, F, Q, K = spec.n_layer, spec.n_embd, spec.n_hidden, spec.q_dim, spec.kv_dim
    shapes = {"attn_norm": (L, W), "ffn_norm": (L, W), "final_norm": (W,), "emb": (spec.vocab, W), "wq": (L, Q, W), "wk": (L, K, W), "wv": (L, K, W), "wo": (L, W, Q), "w1": (L, F, W), "w2": (L, W, F), "w3": (L, F, W)}
    if arch == mf.ARCH_QWEN3:
        shapes.update(q_norm=(L, spec.hd), k_norm=(L, spec.hd))
    w = {k: (1.0 if "norm" in k else 0.0) + rng.standard_normal(s).astype(np.float32) * np.float32(0.05) for k, s in shapes.items()}
    w["emb"][::3] *= np.float32(2.0 ** 70)
    path = str(tmp_path / "overflow.bin")
    mf.write_model_from_weights(path, spec, quant, gs, w)
    eng, o = E.Engine(path, 64), ob.NanoOracle(path, 64)
    assert eng.path.startswith("streaming"), eng.path
    small = np.arange(spec.vocab) % 3 != 0          # (the classifier's rows are the embedding's)
    toks = np.array([4, 6, 7, 9, 12, 5, 8, 10, 3, 11, 13, 15, 2], np.uint32)
    for pos, t in enumerate(toks):
        a, b = eng.forward(int(t), pos), o.forward(int(t), pos)
        if t % 3 == 0:
            assert not a.any() and not b.any(), pos
        elif quant == mf.QUANT_Q4K:
            assert np.isfinite(a).all() and a[small].any(), pos
        else:
            assert np.linalg.norm((a - b)[small]) <= (1e-5 if quant == mf.QUANT_F32 else 2e-2) * np.linalg.norm(b[small]), pos
    eng.close()
    o.close()


# classifiers of warp-owned tiles (32 rows a CTA and more): tiles of 3 rows, of one store of 32 and of more than one, vocabularies that no number of CTAs divides
@pytest.mark.parametrize("quant,gs", [(mf.QUANT_F32, 128), (mf.QUANT_Q80, 64), (mf.QUANT_Q80, 128), (mf.QUANT_Q4K, 128)])
@pytest.mark.parametrize("vocab", [4737, 5003, 71041, 80003])
def test_vocabularies(vocab, quant, gs, monkeypatch):
    monkeypatch.setenv("NB200_STREAM", "1")
    spec = mf.ModelSpec("vocab-%d-%d" % (vocab, gs), mf.ARCH_QWEN3, 64, vocab, 1, 256, 4, 2, 256, 64)
    path = mf.cached_model(spec, quant, gs)
    eng, o = E.Engine(path, 8), ob.NanoOracle(path, 8)
    assert eng.path.startswith("streaming"), eng.path
    for pos, t in enumerate((5, vocab - 1, 3000)):
        a, b = eng.forward(t, pos), o.forward(t, pos)
        assert np.array_equal(a, eng.read(E.F_LOGITS, vocab))          # pinned memory and device, every row of both
        # as above; Q4K: one layer, whose 4-bit activations re-round where a sum changes in its last place
        assert np.linalg.norm(a - b) <= {mf.QUANT_F32: 1e-5, mf.QUANT_Q80: 1e-2, mf.QUANT_Q4K: 0.15}[quant] * np.linalg.norm(b), pos
        assert np.abs(a - b).max() <= (0.01 if quant != mf.QUANT_Q4K else 0.5) * np.abs(b).max(), pos          # no row is lost or another's
    ids = np.zeros(6, np.uint32)
    ids[:3] = 5, vocab - 1, 3000
    assert eng.next_greedy(ids, 2, 0) == int(np.argmax(a))
    eng.close()
    o.close()
