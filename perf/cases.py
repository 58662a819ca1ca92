"""What users have this library do, as measurable cases: decoding, prefill, whole requests, speculative decoding and the
multi-head latent attention step, through the public entry points (``velox_b200.engine.Engine`` and the C ABI).

Kinds of case, one pass each:

  decode   ``batch`` sequences with contexts spread over [lo, hi] tokens generate ``steps`` tokens each; the tokens feed back
           on the device (``Engine.decode``), then the host reads every sequence's tokens and last logits.  ``sample``: top-p
           sampling (0.8 / 0.95) in place of the greedy choice
  stream   one sequence driven from the host, token by token (``Engine.forward_step``: an interactive server that looks at
           every token), then the last logits
  prefill  a prompt of ``lo`` tokens goes through the model; its first token and logits are read
  request  prefill and ``steps`` generated tokens, the whole of a user's call
  spec     prompt-lookup speculative decoding of ``steps`` tokens after a prompt of ``lo`` tokens
  mla      one decode step of a weight-absorbed multi-head latent attention layer: queries into the latent space, the step's
           rows appended, attention over ``batch`` latent caches of [lo, hi] rows, contexts back to the heads' value space

Weights are drawn from the seed.  A trained model's next-token distribution is peaked, while independent random matrices
give nearly flat logits whose greedy choice is a matter of the last bit.  So the head holds the embedding of each token's
predecessor (tokens cycle inside blocks of 16; a tied head repeats the token), and the projections that write the
residual stream are scaled by 1/sqrt(2 * layers), as at the start of training, so that what the embedding put into the
stream is still found there at the end.  Text that comes round again is also what prompt-lookup drafting lives on.
"""
import ctypes as C
import math

import numpy as np
import torch

from velox_b200 import lib as L
from velox_b200 import modelspec as M
from velox_b200.engine import Engine

#: model -> its shape; format -> how linear layers, head and embedding table are stored.
MODELS = {"smollm-135m": M.SMOLLM_135M, "llama3-8b": M.LLAMA3_8B_INT4, "qwen2.5-7b": M.QWEN25_7B_INT8, "qwen2-72b": M.QWEN2_72B_INT4}
FORMATS = {
    "f32": (L.FMT_F32, L.FMT_F32, L.FMT_F32),
    "f16": (L.FMT_F16, L.FMT_F16, L.FMT_F16),
    "bf16": (L.FMT_BF16, L.FMT_BF16, L.FMT_BF16),
    "q4_0": (L.FMT_Q4G64REF, L.FMT_Q4G64REF, L.FMT_Q4G64REF),  # the compiler's own --quantize q4_0
    "q4g32": (L.FMT_Q4G32, L.FMT_Q4G32, L.FMT_F16),
    "i8": (L.FMT_I8PC, L.FMT_I8PC, L.FMT_F16),
}
WEIGHT_BYTES = {L.FMT_F32: 4.0, L.FMT_F16: 2.0, L.FMT_BF16: 2.0, L.FMT_Q4G64REF: 0.5625, L.FMT_Q4G32: 0.5625, L.FMT_I8PC: 1.0}

DRAFT = 4                     # tokens drafted at most per speculative pass
NOPE, ROPE, LATENT, VDIM = 128, 64, 512, 128
ROW = LATENT + ROPE           # one cached token of the latent attention


def engine_case(name, kind, model, fmt, batch=1, lo=512, hi=None, steps=1, sample=False):
    return {"name": name, "kind": kind, "model": model, "fmt": fmt, "batch": batch, "lo": lo, "hi": hi or lo, "steps": steps, "sample": sample}


def mla_case(name, batch, lo, hi, heads=128):
    return {"name": name, "kind": "mla", "batch": batch, "lo": lo, "hi": hi, "heads": heads}


def listed():
    return [
        # the smallest model, uncompressed, one interactive user: launches and latency are all there is
        engine_case("smollm f32 stream", "stream", "smollm-135m", "f32", lo=128, steps=16),
        # the same model as the compiler's own 4-bit format stores it, generating on its own
        engine_case("smollm q4_0 decode", "decode", "smollm-135m", "q4_0", lo=500, steps=32),
        # the headline: one user of an 8B model with 4-bit weights
        engine_case("llama int4 decode", "decode", "llama3-8b", "q4g32", lo=512, steps=16),
        # a long document in that user's context, driven from the host
        engine_case("llama int4 long stream", "stream", "llama3-8b", "q4g32", lo=7900, steps=4),
        # a handful of users on one GPU, sampling
        engine_case("llama int4 batch 4", "decode", "llama3-8b", "q4g32", batch=4, lo=200, hi=3000, steps=8, sample=True),
        # the 8B model in the compiler's own 4-bit format: what its users have on disk
        engine_case("llama q4_0 stream", "stream", "llama3-8b", "q4_0", lo=700, steps=4),
        # a served batch of uneven conversations on 8-bit weights
        engine_case("qwen int8 batch 32", "decode", "qwen2.5-7b", "i8", batch=32, lo=256, hi=2048, steps=8),
        # time to the first token: an ordinary prompt, and a ragged long one on 8-bit weights
        engine_case("llama int4 prefill", "prefill", "llama3-8b", "q4g32", lo=512),
        engine_case("qwen int8 prefill", "prefill", "qwen2.5-7b", "i8", lo=1999),
        # the largest model one GPU holds: a short request, answered
        engine_case("72b int4 request", "request", "qwen2-72b", "q4g32", lo=120, steps=6),
        # text that repeats itself, drafted from the prompt
        engine_case("llama int4 speculative", "spec", "llama3-8b", "q4g32", lo=40, steps=64),
        # the latent-attention layer of a large mixture model, a full batch of long contexts
        mla_case("latent attention batch 64", 64, 1024, 8192),
    ]


def log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(("stream", "decode", "decode", "decode", "prefill", "prefill", "request", "spec", "mla", "mla"))
    if kind == "mla":
        heads = rng.choice((128, 128, 128, 64, 16))  # all heads, or a tensor-parallel rank's share of them
        hi = log_int(rng, 64, 12000)
        batch = log_int(rng, 1, max(1, min(128, 520000 // hi)))
        c = mla_case("", batch, max(1, int(hi * rng.uniform(0.1, 1.0))), hi, heads)
    else:
        model, fmt = rng.choice((("smollm-135m", "f32"), ("smollm-135m", "f16"), ("smollm-135m", "q4_0"), ("llama3-8b", "q4g32"), ("llama3-8b", "q4g32"),
                                 ("llama3-8b", "q4g32"), ("llama3-8b", "q4_0"), ("llama3-8b", "f16"), ("llama3-8b", "bf16"), ("qwen2.5-7b", "i8"),
                                 ("qwen2.5-7b", "i8")))
        if kind == "decode":
            batch = log_int(rng, 1, 32)
            hi = log_int(rng, 16, min(8000, 40000 // batch))
            c = engine_case("", kind, model, fmt, batch, max(1, int(hi * rng.uniform(0.1, 1.0))), hi, min(rng.randint(4, 8), max(1, 64 // batch)), rng.random() < 0.3)
        elif kind == "stream":
            c = engine_case("", kind, model, fmt, lo=log_int(rng, 4, 8000), steps=rng.randint(2, 8))
        elif kind == "prefill":
            c = engine_case("", kind, model, fmt, lo=log_int(rng, 4, 3000))
        elif kind == "request":
            if rng.random() < 0.25:
                c = engine_case("", kind, "qwen2-72b", "q4g32", lo=log_int(rng, 8, 110), steps=rng.randint(1, 6))
            else:
                c = engine_case("", kind, model, fmt, lo=log_int(rng, 8, 1500), steps=rng.randint(2, 16))
        else:
            c = engine_case("", kind, model, fmt, lo=log_int(rng, 8, 400), steps=rng.randint(16, 40))
    del c["name"]
    return c


def lengths(case):
    """Context lengths of a batch: spread over [lo, hi] in an order of no pattern (golden-ratio steps)."""
    lo, hi = case["lo"], case["hi"]
    return [lo + int((hi - lo) * ((0.5 + i * 0.6180339887) % 1.0)) for i in range(case["batch"])]


def spec_of(case):
    w, head, emb = FORMATS[case["fmt"]]
    return MODELS[case["model"]].scaled(name="%s-%s" % (case["model"], case["fmt"]), weight_fmt=w, head_fmt=head, embed_fmt=emb)


def load_weights(eng, spec, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    table = torch.randn((spec.vocab, spec.d_model), device="cuda", dtype=torch.float16, generator=g)
    if spec.tied_lm_head:
        table *= 0.1
    for role, layer, rows, cols, mean, std in spec.tensors():
        if role in (L.ROLE_EMBED, L.ROLE_LM_HEAD):
            t = table if role == L.ROLE_EMBED else (table.view(-1, 16, cols).roll(1, 1) * 0.02).reshape(rows, cols)
            torch.cuda.synchronize()  # the library works on a stream of its own
            L.check(L.load().vb_load_tensor(eng.h, role, layer, C.c_void_p(t.data_ptr()), L.FMT_F16, L.LOC_DEVICE, rows, cols))
            continue
        if role in (L.ROLE_WO, L.ROLE_WDOWN):
            std /= math.sqrt(2 * spec.n_layers)
        L.check(L.load().vb_load_tensor_synthetic(eng.h, role, layer, seed, M.stream_of(role, layer), mean, std, rows, cols))


def prepare_engine(case, seed):
    """A server's state: weights loaded, every sequence's context in the cache, the decode step captured."""
    spec, kind, lens = spec_of(case), case["kind"], lengths(case)
    room = max(lens) + case["steps"] + 16
    eng = Engine(spec, max_seq_len=room, max_batch=case["batch"], lean_weights=case["model"] == "qwen2-72b")
    load_weights(eng, spec, seed)
    if case["sample"]:
        eng.set_sampling(0.8, 0.95, seed=seed)
    prompts = [np.random.default_rng([seed, slot]).integers(0, spec.vocab, size=n).astype(np.uint32) for slot, n in enumerate(lens)]
    for slot in range(case["batch"]):
        eng.reserve(slot, room)
    state = {"case": case, "eng": eng, "prompts": prompts, "lens": lens}
    if kind in ("decode", "stream"):
        for slot, p in enumerate(prompts):
            eng.prefill(p, slot)
        state["next"] = [eng.state(slot)[0] for slot in range(case["batch"])]
    if kind != "prefill":
        eng.build_graph()
    eng.sync()
    return state


def prepare_mla(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    b, h, lens = case["batch"], case["heads"], lengths(case)
    cap = max(lens) + 1

    def normal(*shape, dtype=torch.float32):
        return torch.randn(shape, device="cuda", dtype=dtype, generator=g)

    need = L.load().vb_op_mla_decode_scratch_bytes(b, h, cap, 0)
    return {
        "case": case, "cap": cap, "need": need,
        "cache": normal(b, cap, ROW, dtype=torch.bfloat16),
        "w_uk": normal(h, NOPE, LATENT, dtype=torch.bfloat16) * 0.02, "w_uv": normal(h, VDIM, LATENT, dtype=torch.bfloat16) * 0.02,
        "q_nope": normal(b, h, NOPE), "q_rope": normal(b, h, ROPE), "rows": normal(b, ROW),
        "pos": torch.tensor(lens, device="cuda", dtype=torch.int32), "ctx_len": torch.tensor(lens, device="cuda", dtype=torch.int32) + 1,
        "absorbed": torch.empty((b, h, LATENT), device="cuda"), "q": torch.empty((b, h, ROW), device="cuda"),
        "latent": torch.empty((b, h, LATENT), device="cuda"), "out": torch.empty((b, h, VDIM), device="cuda"),
        "scratch": torch.empty(need, device="cuda", dtype=torch.uint8),
    }


def prepare(case, seed):
    return prepare_mla(case, seed) if case["kind"] == "mla" else prepare_engine(case, seed)


def run_mla(s):
    lib, b, h = L.load(), s["case"]["batch"], s["case"]["heads"]
    stream = C.c_void_p(torch.cuda.current_stream().cuda_stream)

    def ptr(name):
        return C.c_void_p(s[name].data_ptr())

    L.check(lib.vb_op_mla_head_product(ptr("absorbed"), ptr("q_nope"), ptr("w_uk"), h, NOPE, LATENT, b, 0, stream))
    s["q"][:, :, :LATENT] = s["absorbed"]
    s["q"][:, :, LATENT:] = s["q_rope"]
    L.check(lib.vb_op_mla_latent_append(ptr("cache"), ptr("rows"), ptr("pos"), b, s["cap"], stream))
    L.check(lib.vb_op_mla_decode(ptr("latent"), ptr("q"), ptr("cache"), ptr("ctx_len"), b, h, s["cap"], s["cap"], 1.0 / math.sqrt(NOPE + ROPE), 0,
                                 ptr("scratch"), s["need"], stream))
    L.check(lib.vb_op_mla_head_product(ptr("out"), ptr("latent"), ptr("w_uv"), h, LATENT, VDIM, b, 1, stream))
    return {"out": s["out"], "latent": s["latent"], "cache": s["cache"]}


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "mla":
        return run_mla(s)
    eng, steps, batch = s["eng"], case["steps"], case["batch"]
    if kind == "stream":
        tok, pos, tokens = s["next"][0], s["lens"][0], []
        for _ in range(steps):
            tok = eng.forward_step(tok, pos)
            tokens.append(tok)
            pos += 1
        return {"tokens": np.array(tokens, dtype=np.int64), "logits": eng.logits()}
    if kind == "spec":
        tokens, _ = eng.generate_speculative(s["prompts"][0], steps, max_draft_len=DRAFT)
        return {"tokens": tokens.astype(np.int64)}
    if kind == "decode":
        for slot in range(batch):
            eng.set_state(slot, s["next"][slot], s["lens"][slot])
        first = s["lens"]
    else:
        eng.prefill(s["prompts"][0])
        first = [case["lo"] - 1]
        if kind == "request" and steps > 1:
            eng.decode(steps - 1)
    if kind == "decode":
        eng.decode(steps)
    tokens = np.stack([eng.read_tokens(slot, first[slot], steps) for slot in range(batch)]).astype(np.int64)
    return {"tokens": tokens, "logits": np.stack([eng.logits(slot) for slot in range(batch)])}


def work(case):
    lens = lengths(case)
    if case["kind"] == "mla":
        b, h, rows = case["batch"], case["heads"], sum(n + 1 for n in lens)
        products = h * (NOPE + VDIM) * LATENT
        return {"bytes": 2 * rows * ROW + 2 * products + 4 * b * h * (NOPE + ROPE + LATENT + VDIM) + 6 * b * ROW,
                "flops": 2 * rows * h * (ROW + LATENT) + 2 * b * products}
    s = spec_of(case)
    layer = s.d_model * (s.qdim + 2 * s.kvdim) + s.qdim * s.d_model + 3 * s.ffn_dim * s.d_model
    layers, head = layer * s.n_layers, s.vocab * s.d_model
    w_bytes = layers * WEIGHT_BYTES[s.weight_fmt] + head * WEIGHT_BYTES[s.head_fmt]
    kv_row = 4 * s.kvdim * s.n_layers  # K and V of one token, fp16, all layers
    steps, total = case["steps"], {"bytes": 0.0, "flops": 0.0}

    def add(passes, rows, heads, read_rows, pair_sum):
        """`passes` over the weights, `rows` tokens in all, `heads` of them through the head; cache rows read; (query, key) pairs."""
        total["bytes"] += passes * w_bytes + kv_row * (read_rows + rows) + 4 * heads * s.vocab
        total["flops"] += 2 * rows * layers + 2 * heads * head + 4 * pair_sum * s.qdim * s.n_layers

    if case["kind"] in ("prefill", "request", "spec"):
        n = case["lo"]
        add(1, n, 1, n, n * (n + 1) // 2)
    if case["kind"] in ("decode", "stream"):
        pairs = sum(steps * n + steps * (steps + 1) // 2 for n in lens)
        add(steps, steps * len(lens), steps * len(lens), pairs, pairs)
    elif case["kind"] == "request":
        pairs = (steps - 1) * case["lo"] + (steps - 1) * steps // 2
        add(steps - 1, steps - 1, steps - 1, pairs, pairs)
    elif case["kind"] == "spec":
        passes = -(-(steps - 1) // (DRAFT + 1))
        pairs = passes * case["lo"] + passes * (steps + 1) // 2
        add(passes, steps - 1, steps - 1, pairs, pairs * (DRAFT + 1))
    return total


def tolerance(case):
    if case["kind"] == "mla":  # products on bf16 operands; the appended rows are the same bytes
        return {"rel": 1e-2, "max": 0.1}
    # logits behind an fp16 cache and fp16 operands, 2^-11 each, amplified about threefold by the depth of the model
    # (measured against fp32); the tokens are whole numbers and stay what they are
    return {"rel": 5e-3, "max": 0.05}
