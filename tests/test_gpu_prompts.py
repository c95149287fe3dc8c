"""Prompts of model files in portions (csrc/prefill.cu): the K and V rows and the next logits against the same positions one call at a time, at the
edges of the kernels' tiles (64 and 128 positions, 1024 to a portion, rows of weights that no tile of 128 divides, depths that no stage of 128 divides) and
for every group size.

Bounds.  The rows of layer 0 come from the same activation codes (Q80) or exact products (F32): 32-bit sums in another order,
2e-6 of a row's norm.  Deeper Q80 rows and the logits: a change in the last place turns a code here and there, which settles at 1 to
2 % after two to four layers whatever its size; 4e-2.  F32 logits: 1e-5."""
import dataclasses

import numpy as np
import pytest
import torch

from nano_b200 import engine as E, modelfile as mf

pytestmark = pytest.mark.gpu


def rel(a, b):
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


def rows(eng, spec, layer, pos):
    return np.concatenate([eng.read(E.F_KROW, spec.kv_dim, layer, pos), eng.read(E.F_VROW, spec.kv_dim, layer, pos)])


CASES = [("toy-nano", mf.QUANT_F32, 128), ("toy-qwen3", mf.QUANT_F32, 128), ("toy-nano", mf.QUANT_Q80, 32), ("toy-qwen3", mf.QUANT_Q80, 64), ("toy-nano", mf.QUANT_Q80, 128), ("toy-nano", mf.QUANT_Q80, 256),
         ("mini-qwen3", mf.QUANT_Q80, 128), ("mini-nano", mf.QUANT_F32, 128), ("toy-nano-odd", mf.QUANT_F32, 128),
         ("mini-qwen3", mf.QUANT_F32, 128), ("long-qwen3", mf.QUANT_Q80, 128)]
# prompts of m tokens are portions of m - 1: around 64, 128 and 256; past 1024; and, 48 tiles of weight rows and more, where tiles of 128 positions leave no SM
# without a block (from 385 positions for W1|W3, 513 for Q|K|V), the last of them with 1, 2, 64 or all of its positions
LENGTHS = {"toy-qwen3": (34, 64, 1025, 1154), "long-qwen3": (386, 387, 449, 513, 642)}


def check(spec, quant, gs, lengths, room=1200):
    check_file(mf.cached_model(spec, quant, gs), spec, quant, lengths, room)


def check_file(path, spec, quant, lengths, room):
    """Prompts of these lengths in portions against the same positions one call at a time."""
    eng = E.Engine(path, room)
    toks = mf.teacher_tokens(max(1160, *lengths), spec.vocab)
    n = max(lengths)
    last, want, keep = spec.n_layer - 1, {}, {}
    for p in range(n):
        eng.forward_nolog(int(toks[p]), p)
        if p + 1 in lengths:
            want[p + 1] = eng.logits()
    at = lambda m: (0, 1, m // 2, m - 2)          # noqa: E731
    for m in lengths:
        for p in at(m):
            keep[p] = [rows(eng, spec, l, p) for l in (0, last)]
    tol = 1e-5 if quant == mf.QUANT_F32 else 4e-2
    for m in lengths:
        ids = np.zeros(max(m, 33) + 2, np.uint32)
        ids[:33] = toks[:33][::-1]
        eng.decode_greedy(ids, 33, 34)          # leaves rows of another prompt behind
        ids[:m] = toks[:m]
        eng.decode_greedy(ids, m, m + 1)
        assert rel(eng.logits(), want[m]) < tol, m
        for p in at(m):
            assert rel(rows(eng, spec, 0, p), keep[p][0]) < 2e-6, (m, p)
            assert rel(rows(eng, spec, last, p), keep[p][1]) < tol, (m, p)
    eng.close()


@pytest.mark.parametrize("name,quant,gs", CASES)
def test_portions_against_single_positions(name, quant, gs):
    check(dataclasses.replace(mf.PRESETS[name], name=name + "-prompts", block_size=2048), quant, gs, LENGTHS.get(name, (33, 65, 129, 130, 257)))


@pytest.mark.parametrize("width,ff,gs", [(1088, 2240, 32), (1088, 2240, 64), (544, 1120, 32), (320, 4160, 64)])
def test_depths_that_no_stage_of_128_divides(width, ff, gs):
    """The last stage of a depth is a short one, and where 2, 4 or 8 blocks share the depth the last of them may have none (9 stages over 4 blocks, 18 over 8)."""
    spec = mf.ModelSpec("prompts-%d-%d" % (width, ff), mf.ARCH_NANO, 2048, 512, 2, width, 8 if width == 544 else 16, 8, ff)
    check(spec, mf.QUANT_Q80, gs, (10, 65, 66, 130), 400)


def test_penalty_sees_the_prompt_and_short_prompts_stay_as_they_were():
    spec = dataclasses.replace(mf.PRESETS["toy-nano"], name="toy-nano-prompts", block_size=2048)
    path = mf.cached_model(spec, mf.QUANT_F32, 128, cls_gain=4.0)
    eng = E.Engine(path, 200)
    toks = mf.teacher_tokens(64, spec.vocab)
    for n in (20, 64):
        a = np.zeros(101, np.uint32)
        a[:n] = toks[:n]
        b = a.copy()
        for pos in range(99):
            a[pos + 1] = eng.next_greedy(a, pos, 1 if pos < n - 1 else 0, 1.3)
        eng.decode_greedy(b, n, 100, 1.3)
        assert a[:100].tolist() == b[:100].tolist(), n
    eng.close()


@pytest.mark.parametrize("n", [2, 9, 10, 33, 130])
def test_a_call_that_decodes_nothing_leaves_the_last_prompt_position(n):
    spec = dataclasses.replace(mf.PRESETS["toy-nano"], name="toy-nano-prompts", block_size=2048)
    eng = E.Engine(mf.cached_model(spec, mf.QUANT_F32, 128), 200)
    ids = mf.teacher_tokens(n, spec.vocab).astype(np.uint32)
    for p in range(n - 1):
        eng.forward_nolog(int(ids[p]), p)
    want = eng.logits()          # (the streaming path keeps no residual vector that could be read)
    eng.forward_nolog(3, 150)
    eng.decode_greedy(ids.copy(), n, n)
    assert rel(eng.logits(), want) < 1e-5
    eng.close()


def test_a_smaller_model_opened_later_leaves_the_larger_one_working():
    """The limit of dynamic shared memory belongs to a kernel, not to an engine."""
    big = E.Engine(mf.cached_model(dataclasses.replace(mf.PRESETS["mini-nano"], name="mini-nano-two", block_size=2048), mf.QUANT_F32, 128), 600)
    ids = np.zeros(60, np.uint32)
    ids[:40] = mf.teacher_tokens(40, 512)
    want = ids.copy()
    big.decode_greedy(want, 40, 60)
    small = E.Engine(mf.cached_model(dataclasses.replace(mf.PRESETS["toy-nano"], name="toy-nano-two", block_size=2048), mf.QUANT_F32, 128), 100)
    got = ids.copy()
    big.decode_greedy(got, 40, 60)
    assert got.tolist() == want.tolist()
    small.close()
    big.close()


@pytest.mark.parametrize("ff", [12256, 12288, 12320])
def test_rows_around_the_shared_memory_that_needs_no_asking(ff):
    """A 32-bit row of 12288 hidden units (Qwen3-8B's) is 48 KB, to which a kernel's static shared memory comes on top."""
    check(mf.ModelSpec("prompts-64-%d" % ff, mf.ARCH_NANO, 512, 512, 2, 64, 2, 2, ff), mf.QUANT_F32, 128, (10, 65), 200)


def test_a_wide_range_inside_a_matrix_and_a_row(tmp_path):
    """One hidden unit is 2^30 times the others and its outgoing weights 2^-30 times: the same model, number for number in fp32, and portions must not lose
    the small numbers beside the large ones (bounds as above)."""
    spec = dataclasses.replace(mf.PRESETS["toy-nano"], name="range-prompts", block_size=512)
    rng = np.random.default_rng(7)
    L, W, F, Q, K = spec.n_layer, spec.n_embd, spec.n_hidden, spec.q_dim, spec.kv_dim
    shapes = {"attn_norm": (L, W), "ffn_norm": (L, W), "final_norm": (W,), "emb": (spec.vocab, W), "wq": (L, Q, W), "wk": (L, K, W), "wv": (L, K, W), "wo": (L, W, Q), "w1": (L, F, W), "w2": (L, W, F), "w3": (L, F, W)}
    w = {k: (1.0 if "norm" in k else 0.0) + rng.standard_normal(s).astype(np.float32) * np.float32(0.05) for k, s in shapes.items()}
    w["w3"][:, 5] *= np.float32(2.0 ** 30)
    w["w2"][:, :, 5] *= np.float32(2.0 ** -30)
    path = str(tmp_path / "range-prompts.bin")
    mf.write_model_from_weights(path, spec, mf.QUANT_F32, 128, w)
    check_file(path, spec, mf.QUANT_F32, (10, 65, 130), 300)


def small_weights(spec, seed):
    rng = np.random.default_rng(seed)
    L, W, F, Q, K = spec.n_layer, spec.n_embd, spec.n_hidden, spec.q_dim, spec.kv_dim
    shapes = {"attn_norm": (L, W), "ffn_norm": (L, W), "final_norm": (W,), "emb": (spec.vocab, W), "wq": (L, Q, W), "wk": (L, K, W), "wv": (L, K, W), "wo": (L, W, Q), "w1": (L, F, W), "w2": (L, W, F), "w3": (L, F, W)}
    return {k: (1.0 if "norm" in k else 0.0) + rng.standard_normal(s).astype(np.float32) * np.float32(0.05) for k, s in shapes.items()}


def test_keys_that_score_minus_infinity(tmp_path):
    """Forty keys whose score with the last ten queries is below the range of 32 bits, then finite ones: such keys weigh nothing, however many come first."""
    spec = dataclasses.replace(mf.PRESETS["toy-nano"], name="minus-infinity", block_size=512)
    w = small_weights(spec, 3)
    hd = spec.hd
    for h in range(spec.q_dim // hd):          # the last pair of a head turns least: 50 positions leave its sign
        w["wq"][0, h * hd + hd - 2:(h + 1) * hd] = 0.0
        w["wq"][0, h * hd + hd - 1, 1] = 1e20
    for h in range(spec.kv_dim // hd):
        w["wk"][0, h * hd + hd - 2:(h + 1) * hd] = 0.0
        w["wk"][0, h * hd + hd - 1, 0] = -1e20
    w["emb"][:, :2] = 0.0
    w["emb"][:40, 0], w["emb"][40:, 1] = 1.0, 1.0          # tokens below 40 have the keys, the others the queries
    path = str(tmp_path / "minus-infinity.bin")
    mf.write_model_from_weights(path, spec, mf.QUANT_F32, 128, w)
    toks = np.concatenate([np.arange(40), np.arange(60, 70)]).astype(np.uint32)
    eng = E.Engine(path, 100)
    for p, t in enumerate(toks):
        eng.forward_nolog(int(t), p)
    want = [rows(eng, spec, 1, p) for p in range(toks.size - 1)]
    assert np.isfinite(want).all()
    ids = np.zeros(toks.size + 1, np.uint32)
    ids[:-1] = toks
    eng.decode_greedy(ids, toks.size, toks.size + 1)
    for p in (0, 31, 32, 39, 40, 44, 48):
        assert rel(rows(eng, spec, 1, p), want[p]) < 1e-5, p
    eng.close()


@pytest.mark.parametrize("gs", [32, 64, 128, 256])
def test_a_hidden_unit_that_is_not_a_number(gs, tmp_path):
    """A product beyond the range of 32 bits makes one hidden unit of every prompt position minus infinity times zero.  Its activation code is 0 (what the reference's
    conversion gives), in portions as on the path of one kernel per phase."""
    spec = dataclasses.replace(mf.PRESETS["toy-nano"], name="no-number", block_size=512)
    w = small_weights(spec, 4)
    w["emb"][:, 0] = 1.0
    w["w1"][0, 7] = 0.0
    w["w1"][0, 7, 0] = -3e38
    w["w2"][0, :, 7] = 3.0
    path = str(tmp_path / "no-number.bin")
    mf.write_model_from_weights(path, spec, mf.QUANT_Q80, gs, w)
    toks = mf.teacher_tokens(20, spec.vocab).astype(np.uint32)
    ref = E.Engine(path, 100, flags=E.FLAG_NO_STREAM)
    for p, t in enumerate(toks):
        ref.forward_nolog(int(t), p)
    eng = E.Engine(path, 100)
    ids = np.zeros(toks.size + 1, np.uint32)
    ids[:-1] = toks
    eng.decode_greedy(ids, toks.size, toks.size + 1)
    for p in range(toks.size - 1):
        assert rel(rows(eng, spec, 1, p), rows(ref, spec, 1, p)) < 4e-2, p
    eng.close()
    ref.close()


def test_which_prompts_have_the_attention_of_one_kernel():
    """Up to 50 positions (36 where heads are wide or many) a portion's attention is one kernel, above them two, and so it is for the 1, 2 and 3 positions behind 1024 and
    2048 of a longer prompt, whose few queries have more than a thousand keys."""
    spec = dataclasses.replace(mf.PRESETS["toy-qwen3"], name="toy-qwen3-behind", block_size=4096)
    check(spec, mf.QUANT_F32, 128, (37, 38, 51, 52, 1026, 1027, 1028, 2050), 2100)
    wide = dataclasses.replace(mf.PRESETS["mini-qwen3"], name="mini-qwen3-few")
    check(wide, mf.QUANT_F32, 128, (37, 38, 51, 52), 100)

    def launches(s, room, lengths):
        eng, out = E.Engine(mf.cached_model(s, mf.QUANT_F32, 128), room), []
        for m in lengths:
            at = eng.launches
            eng.decode_greedy(np.zeros(m + 2, np.uint32), m + 1, m + 2)
            out.append(eng.launches - at)
        eng.close()
        return out
    a, b, two, c, d, e, four, f = launches(spec, 2100, (50, 51, 1024, 1025, 1026, 1027, 2048, 2049))
    assert a == b - 1 and two == b and c == d == e == four and f - four == four - two          # (a portion of these two layers has one attention)
    a, b, c = launches(wide, 100, (36, 37, 51))
    assert a == b - 3 and b == c


def test_portions_keep_no_copy_of_the_weights():
    """What prompts in portions need beside the model does not grow with its layers: an F32 file opened with them (fast mode) and without (exact mode)."""
    spec = dataclasses.replace(mf.PRESETS["mini-nano"], name="mini-nano-deep", n_layer=12, block_size=512)
    path = mf.cached_model(spec, mf.QUANT_F32, 128)
    used = []
    for flags in (E.FLAG_NO_STREAM | E.FLAG_EXACT, E.FLAG_NO_STREAM | E.FLAG_EXACT, E.FLAG_NO_STREAM):          # (the first: what a first engine loads for good)
        before = torch.cuda.mem_get_info()[0]
        eng = E.Engine(path, 300, flags=flags)
        used.append(before - torch.cuda.mem_get_info()[0])
        eng.close()
    layer = 4 * (spec.q_dim * 2 + 2 * spec.kv_dim + 3 * spec.n_hidden) * spec.n_embd
    assert used[2] - used[1] < 4 * layer, (used, layer)          # one matrix in parts and the activations of a portion; a copy is twelve layers and more
