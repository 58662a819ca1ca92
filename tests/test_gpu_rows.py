"""Products of a few rows of x (mma.sync kernel) and single rows of every format: one decode step of a batch against the
CPU checker, at the sizes where tiles, column groups, weight passes and cluster splits end."""
import functools

import numpy as np
import pytest

import helpers as H
from oracle import oracle as O
from velox_b200 import lib as L
from velox_b200.engine import Engine
from velox_b200.modelspec import LLAMA3_8B_INT4, ModelSpec

pytestmark = pytest.mark.gpu

# 2^-11 of an fp16 cache and of nothing else: logits of N(0, 0.02) heads over unit rows of 512 stay below ~2.5, two layers
TOL = 5e-3
FMTS = {"q4g32": (L.FMT_Q4G32, L.FMT_F16), "q4_0": (L.FMT_Q4G64REF, L.FMT_Q4G64REF), "f16": (L.FMT_F16, L.FMT_F16), "bf16": (L.FMT_BF16, L.FMT_BF16),
        "f32": (L.FMT_F32, L.FMT_F32)}


@pytest.mark.parametrize("fmt", sorted(FMTS))
@pytest.mark.parametrize("batch", [1, 2, 3, 5, 9, 17])
def test_batch_step_matches_checker(fmt, batch):
    w, emb = FMTS[fmt]
    # K of 512 and 1408 (11 blocks of 128: not a multiple of any split), 4112 head rows (257 tiles of 16)
    spec = LLAMA3_8B_INT4.scaled(name="rows-" + fmt, d_model=512, n_layers=2, n_q_heads=8, n_kv_heads=2, head_dim=64, ffn_dim=1408, vocab=4112,
                                 weight_fmt=w, head_fmt=w, embed_fmt=emb)
    eng = H.build_engine(spec, 31, 32, max_batch=batch)
    rng = np.random.default_rng(batch)
    prompts = [rng.integers(0, spec.vocab, size=1 + i % 5).astype(np.uint32) for i in range(batch)]
    toks = rng.integers(0, spec.vocab, size=batch)
    for slot, p in enumerate(prompts):
        eng.reserve(slot, 32)
        eng.prefill(p, slot)
    for slot, p in enumerate(prompts):
        if slot % 4 != 3 or batch < 4:  # every fourth slot sits the step out
            eng.set_state(slot, int(toks[slot]), len(p))
        else:
            eng.set_state(slot, 0, len(p), False)
    eng.decode(1)
    for slot in sorted({0, batch // 2, batch - 1}):
        if slot % 4 == 3 and batch >= 4:
            continue
        ora, _ = H.build_oracle(spec, 31, 32)
        for pos, t in enumerate(prompts[slot]):
            ora.forward_step(int(t), pos)
        ora.forward_step(int(toks[slot]), len(prompts[slot]))
        assert float(np.max(np.abs(eng.logits(slot) - ora.logits))) <= TOL, (fmt, batch, slot)
    eng.close()


@pytest.mark.parametrize("fmt", ["f32", "f16", "bf16", "q4g32", "q4g64ref", "i8pc"])
@pytest.mark.parametrize("in_dim,out_dim,batch", [(64, 1, 1), (64, 7, 2), (576, 33, 1), (1088, 130, 8), (2112, 5, 11), (8192, 19, 4)])
def test_canonical_matvec(vb, oracle, fmt, in_dim, out_dim, batch):
    """Row remainders of the four-row groups, K of whole and ragged steps, passes of eight rows of x."""
    from velox_b200.engine import DeviceBuffer as dev
    c = {"f32": O.FMT_F32, "f16": O.FMT_F16, "bf16": O.FMT_BF16, "q4g32": O.FMT_Q4G32, "q4g64ref": O.FMT_Q4G64REF, "i8pc": O.FMT_I8PC}[fmt]
    w = oracle.fill_normal(out_dim * in_dim, 5, 1, 0.02).reshape(out_dim, in_dim)
    data, scales = oracle.quantize(w, c)
    x = oracle.fill_normal(batch * in_dim, 5, 2, 1.0).reshape(batch, in_dim)
    dw, dx, dy = dev.from_numpy(data), dev.from_numpy(x), dev(batch * out_dim * 4)
    ds = dev.from_numpy(scales) if scales is not None else None
    vb.check(vb.load().vb_op_matmul(dy.ptr, dx.ptr, dw.ptr, ds.ptr if ds else None, c, in_dim, out_dim, batch, None))
    got = dy.to_numpy(np.float32, (batch, out_dim))
    exact = x.astype(np.float64) @ oracle.dequantize(data, scales, c, out_dim, in_dim).astype(np.float64).T
    # fp32 sums of in_dim terms of std 0.02 each: in_dim roundings of 2^-24 of a partial sum below 5 * 0.02 * sqrt(in_dim)
    assert np.max(np.abs(got - exact)) <= in_dim * 2.0 ** -24 * 5 * 0.02 * np.sqrt(in_dim)


@pytest.mark.parametrize("fmt,lean", [("q4g32", False), ("q4g32", True), ("i8", False)])
@pytest.mark.parametrize("n", [9, 17, 33, 34, 65, 66, 129, 140])
def test_prompt_products_from_tensor_memory(fmt, lean, n):
    """Prompts whose n - 1 chunk rows are the edges of the row tiles (8 of 16, 16, 32, 64, 128) and one more, against the CPU checker.
    K of 1024 (split over a cluster), 384 and 1408 / 1472, 576 QKV rows (half a tile over).  Steps at shrinking positions
    look at the cached rows again, each with few others to dilute it."""
    w, ffn = (L.FMT_Q4G32, 1408) if fmt == "q4g32" else (L.FMT_I8PC, 1472)
    spec = LLAMA3_8B_INT4.scaled(name="prompt-" + fmt, d_model=1024, n_layers=2, n_q_heads=12, n_kv_heads=3, head_dim=32, ffn_dim=ffn, vocab=1024,
                                 weight_fmt=w, head_fmt=w)
    eng = Engine(spec, max_seq_len=160, lean_weights=lean)
    eng.load_synthetic(41)
    eng.reserve(0, 160)
    prompt = H.prompt_tokens(spec, 41, n)
    eng.prefill(prompt)
    ora, _ = H.build_oracle(spec, 41, 160)
    for pos, t in enumerate(prompt):
        ora.forward_step(int(t), pos)
    assert float(np.max(np.abs(eng.logits() - ora.logits))) <= TOL
    for pos in (n - 1, n // 2, 16, 2, 1):
        eng.set_state(0, 7, pos)
        eng.decode(1)
        ora.forward_step(7, pos)
        assert float(np.max(np.abs(eng.logits() - ora.logits))) <= TOL, pos
    eng.close()


@pytest.mark.parametrize("head_dim,group", [(32, 2), (64, 3), (128, 1), (128, 8), (256, 2)])
@pytest.mark.parametrize("splits", [1, 3, 7, 11, 16])
def test_attention_slices(head_dim, group, splits):
    """Decode attention cut into any number of slices (odd ones: the merge's slices of the head dimension are uneven), against
    the CPU checker where a slice, a 16-row block or a warp's chunk ends.  Positions shrink: a step overwrites its own row."""
    spec = LLAMA3_8B_INT4.scaled(name="slices", d_model=256, n_layers=2, n_q_heads=2 * group, n_kv_heads=2, head_dim=head_dim, ffn_dim=256, vocab=512,
                                 weight_fmt=L.FMT_F16, head_fmt=L.FMT_F16)
    eng = H.build_engine(spec, 51, 320)
    eng.set_option("attn_splits", splits)
    eng.reserve(0, 320)
    prompt = H.prompt_tokens(spec, 51, 300)
    eng.prefill(prompt)
    ora, _ = H.build_oracle(spec, 51, 320)
    for pos, t in enumerate(prompt):
        ora.forward_step(int(t), pos)
    assert float(np.max(np.abs(eng.logits() - ora.logits))) <= TOL
    for pos in (299, 257, 256, 255, 130, 33, 16, 15, 1, 0):
        eng.set_state(0, 5, pos)
        eng.decode(1)
        ora.forward_step(5, pos)
        assert float(np.max(np.abs(eng.logits() - ora.logits))) <= TOL, pos
    eng.close()


@pytest.mark.parametrize("head_dim", [64, 128])
@pytest.mark.parametrize("n", [449, 514])
def test_long_chunk_attention(head_dim, n):
    """Causal attention of a chunk with blocks for two and for three per SM (40 heads x 7 tiles of 64 rows: 280 blocks, x 9: 360),
    the last tile full or one row long, against the CPU checker; steps at shrinking positions see the second layer's rows."""
    spec = LLAMA3_8B_INT4.scaled(name="chunk", d_model=256, n_layers=2, n_q_heads=40, n_kv_heads=4, head_dim=head_dim, ffn_dim=256, vocab=512,
                                 weight_fmt=L.FMT_F16, head_fmt=L.FMT_F16)
    eng = H.build_engine(spec, 61, 520)
    eng.reserve(0, 520)
    prompt = H.prompt_tokens(spec, 61, n)
    eng.prefill(prompt)
    ora, _ = H.build_oracle(spec, 61, 520)
    for pos, t in enumerate(prompt):
        ora.forward_step(int(t), pos)
    assert float(np.max(np.abs(eng.logits() - ora.logits))) <= TOL
    for pos in (n - 1, 65, 64, 5, 1):
        eng.set_state(0, 5, pos)
        eng.decode(1)
        ora.forward_step(5, pos)
        assert float(np.max(np.abs(eng.logits() - ora.logits))) <= TOL, pos
    eng.close()


def at_offset(dev, a, nbytes):
    """A device copy of `a` that starts nbytes into its allocation: (buffer, address)."""
    buf = dev.from_numpy(np.concatenate([np.zeros(nbytes, np.uint8), np.ascontiguousarray(a).view(np.uint8).reshape(-1)]))
    return buf, buf.ptr.value + nbytes


@pytest.mark.parametrize("fmt", ["f32", "f16", "bf16", "q4g32", "q4g64ref", "i8pc"])
@pytest.mark.parametrize("offset,batch", [(4, 1), (8, 3), (12, 9)])
def test_canonical_matvec_of_rows_at_any_float(vb, oracle, fmt, offset, batch):
    """x and dst may start at any float: same bound as above."""
    from velox_b200.engine import DeviceBuffer as dev
    c = {"f32": O.FMT_F32, "f16": O.FMT_F16, "bf16": O.FMT_BF16, "q4g32": O.FMT_Q4G32, "q4g64ref": O.FMT_Q4G64REF, "i8pc": O.FMT_I8PC}[fmt]
    in_dim, out_dim = 576, 37
    w = oracle.fill_normal(out_dim * in_dim, 6, 1, 0.02).reshape(out_dim, in_dim)
    data, scales = oracle.quantize(w, c)
    x = oracle.fill_normal(batch * in_dim, 6, 2, 1.0).reshape(batch, in_dim)
    dw, ds = dev.from_numpy(data), dev.from_numpy(scales) if scales is not None else None
    (bx, px), (by, py) = at_offset(dev, x, offset), at_offset(dev, np.zeros((batch, out_dim), np.float32), offset)
    vb.check(vb.load().vb_op_matmul(py, px, dw.ptr, ds.ptr if ds else None, c, in_dim, out_dim, batch, None))
    got = by.to_numpy(np.uint8, (offset + batch * out_dim * 4,))[offset:].copy().view(np.float32).reshape(batch, out_dim)
    exact = x.astype(np.float64) @ oracle.dequantize(data, scales, c, out_dim, in_dim).astype(np.float64).T
    assert np.max(np.abs(got - exact)) <= in_dim * 2.0 ** -24 * 5 * 0.02 * np.sqrt(in_dim)


def test_norm_weights_at_any_float(vb):
    """The norm and the rows of a fused instruction from pointers that are 4-byte aligned give what aligned ones give (the same sums)."""
    from velox_b200.engine import DeviceBuffer as dev
    lib, d, ffn = vb.load(), 512, 1024
    rng = np.random.default_rng(3)
    ws = [dev.from_numpy((0.02 * rng.standard_normal(s)).astype(np.float32)) for s in ((d, d), (ffn, d), (ffn, d), (d, ffn))]
    desc = [L.C.byref(L.Weight(w.ptr, None, L.FMT_F32)) for w in ws]
    attn, norm, resid = rng.standard_normal(d).astype(np.float32), (1 + 0.1 * rng.standard_normal(d)).astype(np.float32), rng.standard_normal(d).astype(np.float32)
    scratch, out = dev(ffn * 4), []
    for off in (0, 4):
        (ba, pa), (bn, pn), (bh, ph) = at_offset(dev, attn, off), at_offset(dev, norm, off), at_offset(dev, np.zeros(d, np.float32), off)
        br = dev.from_numpy(resid)
        vb.check(lib.vb_op_fused_outproj_res_swiglu_res(ph, pa, br.ptr, desc[0], pn, desc[1], desc[2], desc[3], d, d, ffn, 1e-5, scratch.ptr, ffn * 4, None))
        out.append(bh.to_numpy(np.uint8, (off + d * 4,))[off:].copy().view(np.float32))
    assert np.array_equal(out[0], out[1])


@pytest.mark.parametrize("fmt", ["f32", "f16", "bf16", "q4g32", "q4g64ref", "i8pc"])
@pytest.mark.parametrize("in_dim,out_dim,batch", [(64, 9, 20), (576, 37, 7), (576, 600, 12), (576, 600, 13), (1088, 130, 17), (576, 4099, 8), (576, 4099, 9), (576, 4099, 13)])
def test_canonical_matvec_passes(vb, oracle, fmt, in_dim, out_dim, batch):
    """Rows of x in passes of one and two (all of them one wave of warps), four, and for fp32 eight; full and ragged last passes."""
    test_canonical_matvec(vb, oracle, fmt, in_dim, out_dim, batch)


class LargeOutput(ModelSpec):
    """The output projections a million times larger: their group scales lie around 1e4, and the last row's logits hang on what the
    second layer's attention finds in the rows before it."""

    def tensors(self):
        return [(r, l, rows, cols, mean, std * 1.5e6 if r == L.ROLE_WO else std) for r, l, rows, cols, mean, std in super().tensors()]


@pytest.mark.parametrize("lean", [False, True])
@pytest.mark.parametrize("n", [12, 30, 70])
def test_prompts_over_int4_scales_beyond_fp16_products(lean, n):
    """(n - 8) * scale beyond 65504: prompts of every route against the CPU checker; a matrix reloaded within range takes the route
    of its new values."""
    base = dict(LLAMA3_8B_INT4.__dict__, name="scales", d_model=512, n_layers=2, n_q_heads=8, n_kv_heads=2, head_dim=64, ffn_dim=1408, vocab=1024)
    for spec in (LargeOutput(**base), ModelSpec(**base)):
        if isinstance(spec, LargeOutput):
            eng = Engine(spec, max_seq_len=96, lean_weights=lean)
            eng.reserve(0, 96)
        eng.spec = spec
        eng.load_synthetic(81)
        prompt = H.prompt_tokens(spec, 81, n)
        eng.prefill(prompt)
        ora, stored = H.build_oracle(spec, 81, 96)
        scales = stored[(L.ROLE_WO, 0)][1].view(np.float16)
        assert (float(np.abs(scales).max()) > 8188) == isinstance(spec, LargeOutput)
        for pos, t in enumerate(prompt):
            ora.forward_step(int(t), pos)
        assert float(np.max(np.abs(eng.logits() - ora.logits))) <= TOL
    eng.close()


@pytest.mark.parametrize("fmt", ["q4_0", "f16", "bf16", "f32"])
@pytest.mark.parametrize("batch", [1, 3, 8])
def test_products_of_a_few_rows_round_like_fp32(oracle, fmt, batch):
    """The head product of a decode step against 64 bits from the same hidden row: x in parts that carry its 24 bits, every 64 of K
    added with a rounding of 2^-24 of the partial sum at most, in random directions: 2^-24 * sqrt(K / 64)."""
    w, emb = FMTS[fmt]
    d = 4096
    spec = LLAMA3_8B_INT4.scaled(name="round-" + fmt, d_model=d, n_layers=1, n_q_heads=4, n_kv_heads=2, head_dim=64, ffn_dim=256, vocab=2048,
                                 weight_fmt=w, head_fmt=w, embed_fmt=emb)
    eng = H.build_engine(spec, 91, 16, max_batch=batch)
    for slot in range(batch):
        eng.reserve(slot, 16)
        eng.prefill(H.prompt_tokens(spec, 91 + slot, 3), slot)
    eng.decode(1)
    data, scales = eng.export_tensor(L.ROLE_LM_HEAD, 0, spec.vocab, d)
    head = O.dequantize(data, scales, w, spec.vocab, d).astype(np.float64)
    nfmt = spec.storage_fmt(L.ROLE_FINAL_NORM)
    norm = O.dequantize(*eng.export_tensor(L.ROLE_FINAL_NORM, 0, 1, d), nfmt, 1, d).astype(np.float64).reshape(d)
    for slot in range(batch):
        x = eng.hidden(slot).astype(np.float64)
        want = head @ (x / np.sqrt((x * x).mean() + spec.rms_eps) * norm)
        assert np.linalg.norm(eng.logits(slot) - want) <= 2.0 ** -24 * np.sqrt(d / 64) * np.linalg.norm(want), slot
    eng.close()


class StrongAttention(ModelSpec):
    """Output projections fifty times larger: what the first layer's attention gives is most of what the second one caches."""

    def tensors(self):
        return [(r, l, rows, cols, mean, std * 50 if r == L.ROLE_WO else std) for r, l, rows, cols, mean, std in super().tensors()]


@pytest.mark.parametrize("head_dim", [64, 128])
@pytest.mark.parametrize("lean,n", [(False, 18), (False, 30), (False, 48), (True, 18), (True, 66)])
def test_short_prompts_keep_the_parts_of_q_and_probabilities(head_dim, lean, n):
    """Prompts that the per-token attention had served give its logits up to the fp16 roundings of the second layer's cache that
    fp32 sums in another order flip (1.6e-5 to 2.6e-5); q and the softmax weights rounded to fp16 are 5.9e-5 to 8.9e-5 off."""
    base = dict(LLAMA3_8B_INT4.__dict__, name="parts", d_model=512, n_layers=2, n_q_heads=8, n_kv_heads=2, head_dim=head_dim, ffn_dim=1408, vocab=1024)
    eng = Engine(StrongAttention(**base), max_seq_len=80, lean_weights=lean)
    eng.load_synthetic(7)
    eng.reserve(0, 80)
    got = []
    for flash in (0, 1):
        eng.set_option("prefill_flash", flash)
        eng.prefill(H.prompt_tokens(eng.spec, 7, n))
        got.append(eng.logits().astype(np.float64))
    eng.close()
    assert np.linalg.norm(got[1] - got[0]) <= 4e-5 * np.linalg.norm(got[0])


@functools.lru_cache(maxsize=1)
def checker_of(fmt, wide):
    """(spec, CPU checker) with rows of 4096: `wide` one layer whose matrices are all large, else two of few heads."""
    w, emb = {**FMTS, "i8": (L.FMT_I8PC, L.FMT_F16)}[fmt]
    kw = dict(n_layers=1, n_q_heads=32, n_kv_heads=8, head_dim=128, ffn_dim=1024, vocab=2048) if wide else dict(
        n_layers=2, n_q_heads=4, n_kv_heads=2, head_dim=64, ffn_dim=1536, vocab=512)
    spec = LLAMA3_8B_INT4.scaled(name="k4096-" + fmt, d_model=4096, weight_fmt=w, head_fmt=w, embed_fmt=emb, **kw)
    return spec, H.build_oracle(spec, 31, 144)[0]


TOL_4096 = TOL * 8 ** 0.5  # rows eight times as long: logits sqrt(8) times as large


@pytest.mark.parametrize("fmt,batch", [("bf16", 3), ("bf16", 4), ("f16", 3), ("f16", 4), ("q4_0", 1), ("q4_0", 3), ("q4_0", 4), ("q4_0", 8),
                                       ("q4g32", 2), ("q4g32", 4), ("q4g32", 8)])
def test_large_matrices_match_checker(fmt, batch):
    """Matrices of 8M weights and more (QKV 6144 x 4096, O 4096 x 4096 onto the residual stream, gate/up 2048 x 4096, head 2048 x 4096):
    one and two groups of eight columns, K split over clusters of 4 and 8, one row of group-64."""
    spec, ora = checker_of(fmt, True)
    eng = H.build_engine(spec, 31, 16, max_batch=batch)
    rng = np.random.default_rng(batch)
    toks = rng.integers(0, spec.vocab, size=(batch, 3))
    for slot in range(batch):
        eng.reserve(slot, 16)
        eng.prefill(toks[slot, :2].astype(np.uint32), slot)
        eng.set_state(slot, int(toks[slot, 2]), 2)
    eng.decode(1)
    for slot in sorted({0, batch // 2, batch - 1}):
        for pos, t in enumerate(toks[slot]):
            ora.forward_step(int(t), pos)
        assert float(np.max(np.abs(eng.logits(slot) - ora.logits))) <= TOL_4096, slot
    eng.close()


@pytest.mark.parametrize("fmt,lean", [("i8", False), ("q4g32", False), ("q4g32", True)])
def test_prompt_products_split_over_large_clusters(fmt, lean):
    """Prompts over rows of 4096: QKV of 512 rows splits K over clusters of 8, gate/up of 3072 over 4; one to 128 rows a tile.  Steps at
    shrinking positions look at the cached rows again, with few others to dilute them."""
    spec, ora = checker_of(fmt, False)
    ns, later = (17, 33, 65, 129), (16, 2, 1)
    prompt, want, steps = H.prompt_tokens(spec, 31, ns[-1]), {}, []
    for pos, t in enumerate(prompt):
        ora.forward_step(int(t), pos)
        if pos + 1 in ns:
            want[pos + 1] = ora.logits.copy()
    for pos in later:
        ora.forward_step(7, pos)
        steps.append(ora.logits.copy())
    eng = Engine(spec, max_seq_len=144, lean_weights=lean)
    eng.load_synthetic(31)
    eng.reserve(0, 144)
    for n in ns:
        eng.prefill(prompt[:n])
        assert float(np.max(np.abs(eng.logits() - want[n]))) <= TOL_4096, n
        for pos, w in zip(later, steps):
            eng.set_state(0, 7, pos)
            eng.decode(1)
            assert float(np.max(np.abs(eng.logits() - w))) <= TOL_4096, (n, pos)
    eng.close()


@pytest.mark.parametrize("fmt,batch", [("q4g32", 2), ("q4g32", 4), ("q4g32", 5), ("q4g32", 8), ("q4g32", 9), ("q4_0", 1), ("q4_0", 2), ("q4_0", 3), ("q4_0", 5)])
@pytest.mark.parametrize("ffn", [4096, 4224, 6272])
def test_few_rows_of_long_and_short_matrices(fmt, batch, ffn):
    """x resident in shared memory (K of 2048 and 4096) and going round a ring of chunks (33 weight blocks: the last pair is one block
    and its chunk one pair; 49: four chunks), one pass of 8 columns, of 16, and a second pass, against the CPU checker."""
    w, emb = FMTS[fmt]
    spec = LLAMA3_8B_INT4.scaled(name="few-" + fmt, d_model=2048, n_layers=1, n_q_heads=16, n_kv_heads=4, head_dim=128, ffn_dim=ffn, vocab=4112,
                                 weight_fmt=w, head_fmt=w, embed_fmt=emb)
    eng = H.build_engine(spec, 71, 32, max_batch=batch)
    toks = np.random.default_rng(batch).integers(0, spec.vocab, size=(batch, 2))
    for slot in range(batch):
        eng.reserve(slot, 32)
        eng.set_state(slot, int(toks[slot, 0]), 0, slot != 1)  # the second slot sits the first step out
    eng.decode(1)
    for slot in range(batch):
        eng.set_state(slot, int(toks[slot, 1]), 1 if slot != 1 else 0)
    eng.decode(1)
    for slot in sorted({0, min(1, batch - 1), batch // 2, batch - 1}):
        ora, _ = H.build_oracle(spec, 71, 32)
        for pos, t in enumerate(toks[slot] if slot != 1 else toks[slot, 1:]):
            ora.forward_step(int(t), pos)
        # rows of 2048: logits up to twice those of the 512 above
        assert float(np.max(np.abs(eng.logits(slot) - ora.logits))) <= 2 * TOL, (slot,)
    eng.close()


@pytest.mark.parametrize("fmt", ["f16", "q4_0", "i8"])
@pytest.mark.parametrize("n", [131, 1001])
def test_gate_and_up_of_a_chunk_by_pairs_of_blocks(fmt, n):
    """SwiGLU tiles of a prompt of two and of eight tiles of 128 rows, all directions ragged."""
    w = L.FMT_I8PC if fmt == "i8" else FMTS[fmt][0]
    spec = LLAMA3_8B_INT4.scaled(name="pairs-" + fmt, d_model=256, n_layers=2, n_q_heads=4, n_kv_heads=2, head_dim=64, ffn_dim=2496, vocab=512,
                                 weight_fmt=w, head_fmt=L.FMT_F16, embed_fmt=L.FMT_F16)
    eng = H.build_engine(spec, 81, 1008)
    eng.reserve(0, 1008)
    prompt = H.prompt_tokens(spec, 81, n)
    eng.prefill(prompt)
    ora, _ = H.build_oracle(spec, 81, 1008)
    for pos, t in enumerate(prompt):
        ora.forward_step(int(t), pos)
    assert float(np.max(np.abs(eng.logits() - ora.logits))) <= TOL
    for pos in (n - 1, 129, 128, 5, 1):
        eng.set_state(0, 5, pos)
        eng.decode(1)
        ora.forward_step(5, pos)
        assert float(np.max(np.abs(eng.logits() - ora.logits))) <= TOL, pos
    eng.close()


@pytest.mark.parametrize("d_model,ffn,batch", [(448, 1184, 3), (512, 20608, 15), (512, 1408, 16), (2048, 4224, 5), (2048, 4224, 9)])
def test_few_int8_rows_on_the_integer_tensor_cores(d_model, ffn, batch):
    """Three byte planes of 16 rows: K that is no multiple of 128, rows beyond what a block keeps in registers, all 16 rows, and models
    whose steps take that way by themselves; one slot sits a step out."""
    spec = LLAMA3_8B_INT4.scaled(name="planes", d_model=d_model, n_layers=2, n_q_heads=d_model // 64, n_kv_heads=1 if d_model == 448 else 2, head_dim=64,
                                 ffn_dim=ffn, vocab=1040, weight_fmt=L.FMT_I8PC, head_fmt=L.FMT_I8PC)
    eng = H.build_engine(spec, 91, 32, max_batch=batch)
    if d_model < 2048:
        eng.set_option("decode_gemm", 1)
    eng.build_graph()  # (makes the workspaces of the step's products, as a prompt does; without them it takes others)
    toks = np.random.default_rng(batch).integers(0, spec.vocab, size=(batch, 2))
    for slot in range(batch):
        eng.reserve(slot, 32)
        eng.set_state(slot, int(toks[slot, 0]), 0, slot != 1)
    eng.decode(1)
    for slot in range(batch):
        eng.set_state(slot, int(toks[slot, 1]), 1 if slot != 1 else 0)
    eng.decode(1)
    for slot in sorted({0, 1, batch // 2, batch - 1}):
        ora, _ = H.build_oracle(spec, 91, 32)
        for pos, t in enumerate(toks[slot] if slot != 1 else toks[slot, 1:]):
            ora.forward_step(int(t), pos)
        # rows of 2048: logits up to twice those of 512
        assert float(np.max(np.abs(eng.logits(slot) - ora.logits))) <= (2 if d_model == 2048 else 1) * TOL, (slot,)
    eng.close()


@pytest.mark.parametrize("d_model,ffn,batch", [(2048, 4224, 5), (2048, 16384, 3), (2048, 16384, 4)])
def test_few_int8_rows_and_the_options_around_them(d_model, ffn, batch):
    """Steps that take the integer tensor cores by themselves: "decode_gemm" 0, the default of such a context, leaves them there (the same
    bits), "few_i8" 0 does not (its matrix-vector products take 16 bits of every 32 values), 1 brings them back."""
    spec = LLAMA3_8B_INT4.scaled(name="few", d_model=d_model, n_layers=1, n_q_heads=16, n_kv_heads=4, head_dim=128, ffn_dim=ffn, vocab=1040,
                                 weight_fmt=L.FMT_I8PC, head_fmt=L.FMT_I8PC)
    eng = H.build_engine(spec, 92, 16, max_batch=batch)
    for slot in range(batch):
        eng.reserve(slot, 16)

    def step():
        eng.build_graph()  # (makes the workspaces of the step's products, as a prompt does)
        for slot in range(batch):
            eng.set_state(slot, 7 * slot + 3, 0)
        before = eng.launch_count()
        eng.decode(1)
        return eng.launch_count() - before, np.stack([eng.logits(slot) for slot in range(batch)])

    launches, want = step()
    eng.set_option("decode_gemm", 0)
    again = step()
    assert again[0] == launches and np.array_equal(again[1], want)
    eng.set_option("few_i8", 0)
    other = step()[1]
    assert not np.array_equal(other, want) and float(np.max(np.abs(other - want))) <= TOL
    eng.set_option("few_i8", 1)
    assert np.array_equal(step()[1], want)
    ora, _ = H.build_oracle(spec, 92, 16)
    ora.forward_step(7 * (batch - 1) + 3, 0)
    assert float(np.max(np.abs(want[-1] - ora.logits))) <= 2 * TOL  # rows of 2048: logits up to twice those of 512
    eng.close()


def bare_int8_engine(d_model, ffn, batch, rows):
    """One int8 layer whose attention adds nothing (Wo = 0), over fp32 embedding rows: (engine, its weights dequantised in 64 bits)."""
    spec = LLAMA3_8B_INT4.scaled(name="bare", d_model=d_model, n_layers=1, n_q_heads=d_model // 64, n_kv_heads=1 if d_model == 448 else 2, head_dim=64,
                                 ffn_dim=ffn, vocab=1040, weight_fmt=L.FMT_I8PC, head_fmt=L.FMT_I8PC, embed_fmt=L.FMT_F32)
    eng = H.build_engine(spec, 93, 16, max_batch=batch)
    eng.load_tensor(L.ROLE_WO, 0, np.zeros((d_model, d_model), np.float32))
    table = np.zeros((spec.vocab, d_model), np.float32)
    table[:len(rows)] = rows
    eng.load_tensor(L.ROLE_EMBED, 0, table)
    eng.set_option("decode_gemm", 1)
    for slot in range(batch):
        eng.reserve(slot, 16)
    w = {}
    for role, n, k in ((L.ROLE_MLP_NORM, 1, d_model), (L.ROLE_FINAL_NORM, 1, d_model), (L.ROLE_WGATE, ffn, d_model), (L.ROLE_WUP, ffn, d_model),
                       (L.ROLE_WDOWN, d_model, ffn), (L.ROLE_LM_HEAD, spec.vocab, d_model)):
        data, scales = eng.export_tensor(role, 0, n, k)
        if spec.storage_fmt(role) == L.FMT_I8PC:
            w[role] = data.astype(np.float64) * scales.view(np.float16).astype(np.float64)[:, None]
        else:
            w[role] = data.view(np.float16).astype(np.float64).reshape(k)
    return spec, eng, w


def bare_step(eng, batch):
    eng.build_graph()
    for slot in range(batch):
        eng.set_state(slot, slot, 0)
    eng.decode(1)
    return np.stack([eng.hidden(slot) for slot in range(batch)]), np.stack([eng.logits(slot) for slot in range(batch)])


@pytest.mark.parametrize("batch", [1, 3, 15, 16, 17, 32])
@pytest.mark.parametrize("d_model,ffn", [(448, 1184), (512, 20608), (1024, 1408)])
def test_int8_products_of_a_batch_against_64_bits(d_model, ffn, batch):
    """SiLU, residual (K split over blocks) and plain products, K that is no multiple of 128 and rows beyond a block's registers; rows with an
    outlier of 1000 and of 100000.  x has 24 bits of its row's largest magnitude m up to 16 rows, 16 bits beyond: rounded to steps of m / P, each
    value is off by m / (P sqrt(12)) rms, a product by that times the norm of the matrix (a plane too few: 256 times as much)."""
    rng = np.random.default_rng(batch)
    rows = rng.standard_normal((batch, d_model)).astype(np.float32)
    for row, outlier in ((batch - 1, 1.0e3), (batch // 2, 1.0e5)):
        if batch > 1:
            rows[row, 5 + row] = outlier
    spec, eng, w = bare_int8_engine(d_model, ffn, batch, rows)
    hidden, logits = bare_step(eng, batch)
    eng.close()
    levels = (8.3e6 if batch <= 16 else 32000.0) * np.sqrt(12.0)
    norm = lambda v, g: v / np.sqrt((v * v).mean() + spec.rms_eps) * g
    gate, up, down, head = w[L.ROLE_WGATE], w[L.ROLE_WUP], w[L.ROLE_WDOWN], w[L.ROLE_LM_HEAD]
    for slot in range(batch):
        e = rows[slot].astype(np.float64)
        x = norm(e, w[L.ROLE_MLP_NORM])
        g, u = gate @ x, up @ x
        sig = 1.0 / (1.0 + np.exp(-g))
        act = g * sig * u
        step = np.abs(x).max() / levels
        off = np.sqrt(((sig * (1 + g * (1 - sig)) * u) ** 2 * (gate ** 2).sum(1) + (g * sig) ** 2 * (up ** 2).sum(1)).sum()) * step  # of act
        fro = np.linalg.norm(down)
        bound = 1.5 * (np.abs(act).max() / levels * fro + (off + 2.0 ** -22 * np.linalg.norm(act)) * fro / np.sqrt(ffn))
        want = e + down @ act
        assert np.linalg.norm(hidden[slot] - want) <= bound + 2.0 ** -24 * np.linalg.norm(want), slot
        x = norm(hidden[slot].astype(np.float64), w[L.ROLE_FINAL_NORM])
        want = head @ x
        assert np.linalg.norm(logits[slot] - want) <= 1.5 * np.abs(x).max() / levels * np.linalg.norm(head) + 2.0 ** -22 * np.linalg.norm(want), slot


@pytest.mark.parametrize("batch", [3, 16, 17, 32])
@pytest.mark.parametrize("d_model,ffn", [(512, 1408), (512, 20608)])
@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
def test_an_int8_row_that_is_not_finite_gives_no_numbers(d_model, ffn, batch, bad):
    rows = np.random.default_rng(7).standard_normal((batch, d_model)).astype(np.float32)
    _, eng, _ = bare_int8_engine(d_model, ffn, batch, rows)
    want = bare_step(eng, batch)
    eng.close()
    rows[1, 77] = bad
    _, eng, _ = bare_int8_engine(d_model, ffn, batch, rows)
    got = bare_step(eng, batch)
    eng.close()
    others = np.arange(batch) != 1
    for a, b in zip(got, want):
        assert np.all(np.isnan(a[1])) and np.array_equal(a[others], b[others])


SLICES = LLAMA3_8B_INT4.scaled(name="slices8", d_model=256, n_layers=1, n_q_heads=32, n_kv_heads=8, head_dim=128, ffn_dim=256, vocab=512,
                               weight_fmt=L.FMT_F16, head_fmt=L.FMT_F16)
SLICE_PROMPTS = (600, 333)


@functools.lru_cache(maxsize=None)
def slices_want(slot):
    n = SLICE_PROMPTS[slot]
    ora, _ = H.build_oracle(SLICES, 52, 640)
    for pos, t in enumerate(H.prompt_tokens(SLICES, 52 + slot, n)):
        ora.forward_step(int(t), pos)
    want = {}
    for pos in (n - 1, 300, 257, 256, 130, 16, 15, 0):
        ora.forward_step(5, pos)
        want[pos] = ora.logits.copy()
    return want


@pytest.mark.parametrize("max_seq", [640, 4500])
@pytest.mark.parametrize("batch", [1, 2])
@pytest.mark.parametrize("splits", [0, 2, 4, 6, 8, 16])
def test_attention_slices_of_many_clusters(splits, batch, max_seq):
    """Eight and sixteen (sequence, KV head) pairs, whose clusters may not all run at once, and block tables on both sides of the 256 entries
    that are fetched whole; 0: the number of slices that the rule takes, more than eight ask for no more than eight here."""
    eng = H.build_engine(SLICES, 52, max_seq, max_batch=batch)
    eng.set_option("attn_splits", splits)
    for slot in range(batch):
        eng.reserve(slot, 640)
        eng.prefill(H.prompt_tokens(SLICES, 52 + slot, SLICE_PROMPTS[slot]), slot)
    for step in range(8):
        at = [list(slices_want(slot))[step] for slot in range(batch)]
        for slot in range(batch):
            eng.set_state(slot, 5, at[slot])
        eng.decode(1)
        for slot in range(batch):
            assert float(np.max(np.abs(eng.logits(slot) - slices_want(slot)[at[slot]]))) <= TOL, (slot, at[slot])
    for bad in (-1, 17):
        with pytest.raises(L.VeloxError):
            eng.set_option("attn_splits", bad)
    eng.close()
