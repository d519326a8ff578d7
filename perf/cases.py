"""The work a user of this backend has it do, as measurable cases: batched decode and chunked prefill of Llama-shaped models
through the compiled executable, and the operators a graph calls one by one.

listed()            the named cases
draw(rng)           one more case of the same ranges
prepare(case, seed) inputs, weights, pages and handles a program holds before the call, made from the seed
run(state)          one pass through the public entry points; returns what the path computes
work(case)          bytes and operations one pass cannot do without
tolerance(case)     how far another correct implementation at the same precision may be off

Weights are ~N(0, 0.02). Q4_0 and Q8_0 come from the library's quantizer; the K-quants, for which it has none, are random
code bytes under block scales that give the same spread around zero. Cached K / V rows and activations are ~N(0, 1).
"""
import math

import numpy as np
import torch

import effect_torch_b200 as et

BLOCK = 16
LLAMA_8B = dict(d_model=4096, q_heads=32, kv_heads=8, head_dim=128, ffn=14336, vocab=128256, rms_eps=1e-5, rope_theta=500000.0)
LLAMA_70B = dict(d_model=8192, q_heads=64, kv_heads=8, head_dim=128, ffn=28672, vocab=128256, rms_eps=1e-5, rope_theta=500000.0)
MODELS = {"8b": LLAMA_8B, "70b": LLAMA_70B}

CODECS = {"q4_0": et.Q4_0, "q8_0": et.Q8_0, "q2_k": et.Q2_K, "q3_k": et.Q3_K, "q4_k": et.Q4_K, "q5_k": et.Q5_K, "q6_k": et.Q6_K}
# codec -> (values per block, bytes per block)
BLOCK_FORMAT = {"q4_0": (32, 18), "q8_0": (32, 34), "q2_k": (256, 84), "q3_k": (256, 110), "q4_k": (256, 144), "q5_k": (256, 176),
                "q6_k": (256, 210)}
# codec -> (byte offset, value) of its f16 block scales, chosen so that random code bytes decode to zero mean and 0.02 spread
K_SCALES = {"q2_k": ((80, 1.44e-3), (82, 2.16e-3)), "q3_k": ((108, 4.7e-4),), "q4_k": ((0, 7.75e-5), (2, 5.81e-4)),
            "q5_k": ((0, 3.8e-5), (2, 5.89e-4)), "q6_k": ((208, 1.46e-5),)}
KV = {"f32": (et.KV_F32, 4), "f16": (et.KV_F16, 2), "bf16": (et.KV_BF16, 2), "u8": (et.KV_U8, 1)}
ROPE = {"half": et.HALF_SPLIT, "pairs": et.INTERLEAVED_PAIRS}
EPILOGUES = {"none": et.EPILOGUE_NONE, "residual": et.EPILOGUE_RESIDUAL, "swiglu": et.EPILOGUE_SWIGLU}


def listed():
    return [
        # The headline workload: the 8B shape, Q4_0, 32 sequences whose 512-token prompts sit in the prefix cache, 16 steps.
        dict(name="decode-8b-q4_0-b32", kind="decode", model="8b", layers=32, weights="q4_0", batch=32, context=512, ragged=False,
             steps=16, kv="f16", read="tokens", rope="half"),
        # One chat user on a mixed K-quant file, a long context, logits read back for sampling on the host.
        dict(name="decode-8b-kmix-b1", kind="decode", model="8b", layers=32, weights="kmix", batch=1, context=3072, ragged=False,
             steps=8, kv="f16", read="logits", rope="pairs"),
        # A small server: 8 sequences of different lengths over the int8 cache, Q8_0 weights.
        dict(name="decode-8b-q8_0-b8-u8", kind="decode", model="8b", layers=8, weights="q8_0", batch=8, context=4096, ragged=True,
             steps=8, kv="u8", read="logits", rope="half"),
        # The 70B shape at batch 64 with contexts up to 8192: attention weighs as much as the projections.
        dict(name="decode-70b-q4_0-b64", kind="decode", model="70b", layers=4, weights="q4_0", batch=64, context=8192, ragged=True,
             steps=8, kv="f16", read="tokens", rope="half"),
        # Prompts of a batch, prefilled in chunks.
        dict(name="prefill-8b-q4_0-b8", kind="prefill", model="8b", layers=32, weights="q4_0", batch=8, prompt=512, chunk=256, kv="f16",
             rope="half"),
        # One prompt of an odd length on a mixed K-quant file: a whole chunk and a ragged rest, bf16 cache.
        dict(name="prefill-8b-kmix-b1", kind="prefill", model="8b", layers=32, weights="kmix", batch=1, prompt=777, chunk=512, kv="bf16",
             rope="pairs"),
        # The reference's CPU-sized f32 model in reference-order arithmetic: prefill and 63 device-resident greedy steps. The
        # smallest launches there are.
        dict(name="exact-tiny-b4", kind="exact", layers=4, d_model=256, q_heads=4, kv_heads=2, head_dim=64, ffn=688, vocab=4096, batch=4,
             prompt=32, steps=63),
        # One token through a run of square projections: latency per call, every weight from HBM.
        dict(name="linear-q4_0-v1", kind="linear", weights="q4_0", rows=4096, columns=4096, vectors=1, calls=8, epilogue="none"),
        # The operator route on raw GGUF rows, which takes every codec.
        dict(name="raw-linear-q4_k-v5", kind="raw", weights="q4_k", rows=14336, columns=4096, vectors=5),
        # The paged-attention microbenchmark: 64 sequences of 128 to 4096 tokens over interleaved pages.
        dict(name="attention-b64", kind="attention", batch=64, q_heads=32, kv_heads=8, head_dim=128, shortest=128, longest=4096, kv="f16"),
        # Stochastic sampling of one decode step's logits with the usual filters.
        dict(name="sample-b32", kind="sample", rows=32, vocab=128256, temperature=0.8, top_k=40, top_p=0.95),
        # Load-time coding of a projection: f32 rows packed, and the packed rows decoded again.
        dict(name="transcode-q4_0", kind="transcode", weights="q4_0", rows=14336, columns=4096),
    ]


def _spread(rng, low, high):
    """A whole number between low and high, even over the logarithm."""
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.choice(["decode", "decode", "prefill", "exact", "linear", "linear", "raw", "attention", "sample", "transcode"])
    if kind == "decode":
        model = rng.choice(["8b", "8b", "70b"])
        batch = _spread(rng, 1, 64)
        longest = min(8192, 131072 // batch)
        steps = rng.randint(6, 15)
        return dict(kind=kind, model=model, layers=rng.randint(2, 4) if model == "70b" else rng.randint(2, 8),
                    weights=rng.choice(["q4_0", "q4_0", "q8_0", "kmix", "q4_k", "q6_k"]), batch=batch,
                    context=_spread(rng, 2, longest // BLOCK) * BLOCK, ragged=rng.random() < 0.5, steps=steps,
                    kv=rng.choice(["f16", "f16", "bf16", "u8"]), read="tokens" if batch * steps >= 256 else "logits",
                    rope=rng.choice(["half", "pairs"]))
    if kind == "prefill":
        batch = _spread(rng, 1, 16)
        chunk = _spread(rng, 16, 2048 // batch)
        return dict(kind=kind, model="8b", layers=rng.randint(2, 8), weights=rng.choice(["q4_0", "q4_0", "q8_0", "kmix", "q5_k"]),
                    batch=batch, prompt=_spread(rng, chunk, 4 * chunk), chunk=chunk, kv=rng.choice(["f16", "f16", "bf16", "u8"]),
                    rope=rng.choice(["half", "pairs"]))
    if kind == "exact":
        head_dim, kv_heads, group = rng.choice([32, 64]), rng.randint(1, 4), rng.choice([1, 2, 4])
        return dict(kind=kind, layers=rng.randint(2, 6), d_model=32 * rng.randint(4, 16), q_heads=kv_heads * group, kv_heads=kv_heads,
                    head_dim=head_dim, ffn=8 * rng.randint(24, 128), vocab=_spread(rng, 256, 8192), batch=rng.randint(1, 8),
                    prompt=rng.randint(2, 64), steps=rng.randint(16, 80))
    if kind == "linear":
        weights = rng.choice(["q4_0", "q8_0", "q3_k", "q4_k", "q5_k", "q6_k"])
        rows, columns = _spread(rng, 64, 1792) * 16, _spread(rng, 4, 56) * 256
        return dict(kind=kind, weights=weights, rows=rows, columns=columns, vectors=_spread(rng, 1, 1024),
                    calls=max(1, min(8, int(3e8 / (rows * columns)))), epilogue=rng.choice(["none", "residual", "swiglu"]))
    if kind == "raw":
        weights = rng.choice(sorted(CODECS))
        return dict(kind=kind, weights=weights, rows=_spread(rng, 256, 16384), columns=256 * _spread(rng, 4, 32), vectors=_spread(rng, 1, 32))
    if kind == "attention":
        kv_heads = rng.choice([1, 2, 4, 8])
        batch = _spread(rng, 1, 64)
        longest = _spread(rng, 64, 4096)
        return dict(kind=kind, batch=batch, q_heads=kv_heads * rng.choice([1, 2, 4, 8]), kv_heads=kv_heads, head_dim=rng.choice([64, 128]),
                    shortest=rng.randint(1, longest), longest=longest, kv=rng.choice(["f16", "f16", "bf16", "u8"]))
    if kind == "sample":
        vocab = _spread(rng, 2000, 131072)
        return dict(kind=kind, rows=_spread(rng, 1, 64), vocab=vocab, temperature=rng.choice([0.0, 0.6, 0.8, 1.0, 1.3]),
                    top_k=rng.choice([0, 0, 20, 40, 200]), top_p=rng.choice([1.0, 0.9, 0.95]))
    weights = rng.choice(["q4_0", "q4_0", "q8_0", "q8_0", "q4_k", "q6_k"])
    return dict(kind="transcode", weights=weights, rows=_spread(rng, 16, 16384), columns=256 * _spread(rng, 2, 16))


# ---------------------------------------------------------------------------------------------- building blocks
_runtime = None


def runtime():
    """The process's one runtime, as a server keeps it."""
    global _runtime
    if _runtime is None:
        _runtime = et.Runtime(0)
    return _runtime


def _generator(seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(int(seed) * 7919 + 17)
    return gen


def _row_bytes(codec, columns):
    values, size = BLOCK_FORMAT[codec]
    return columns // values * size


def _packed(gen, codec, rows, columns):
    """[rows, row bytes] u8 of a projection in the codec's file layout, on the device."""
    rt = runtime()
    if codec in K_SCALES:
        packed = torch.randint(0, 256, (rows, columns // 256, BLOCK_FORMAT[codec][1]), generator=gen, device="cuda", dtype=torch.uint8)
        for offset, value in K_SCALES[codec]:
            packed[:, :, offset:offset + 2] = torch.tensor([value], dtype=torch.float16).view(torch.uint8).cuda()
        torch.cuda.synchronize()
        return packed.view(rows, -1)
    packed = torch.empty((rows, _row_bytes(codec, columns)), dtype=torch.uint8, device="cuda")
    for r0 in range(0, rows, 32768):
        r1 = min(rows, r0 + 32768)
        w = torch.randn((r1 - r0, columns), generator=gen, device="cuda").mul_(0.02)
        torch.cuda.synchronize()
        rt.quantize_into(CODECS[codec], w, r1 - r0, columns, packed[r0:r1])
        rt.synchronize()
    return packed


def _geometry(case):
    if case["kind"] == "exact":
        g = {k: case[k] for k in ("d_model", "q_heads", "kv_heads", "head_dim", "ffn", "vocab")}
        return dict(g, rms_eps=1e-5, rope_theta=10000.0, layers=case["layers"])
    return dict(MODELS[case["model"]], layers=case["layers"])


def _projections(case):
    """(slot, layer, rows, columns, codec) of every matrix a decode step multiplies by."""
    g = _geometry(case)
    d, qw, kvw, ffn = g["d_model"], g["q_heads"] * g["head_dim"], g["kv_heads"] * g["head_dim"], g["ffn"]
    slots = ((et.W_Q, qw, d), (et.W_K, kvw, d), (et.W_V, kvw, d), (et.W_O, d, qw), (et.W_GATE, ffn, d), (et.W_UP, ffn, d), (et.W_DOWN, d, ffn))
    weights = "f32" if case["kind"] == "exact" else case["weights"]
    for layer in range(g["layers"]):
        for slot, rows, columns in slots:
            codec = weights
            if weights == "kmix":  # the usual mixed recipe: v and down of every other layer, and the head, at more bits
                codec = "q6_k" if layer % 2 == 0 and slot in (et.W_V, et.W_DOWN) else "q4_k"
            yield slot, layer, rows, columns, codec
    yield et.W_HEAD, 0, g["vocab"], d, "q6_k" if weights == "kmix" else weights


def _model(case, gen, batch, max_tokens, kv, max_advance, rope=et.HALF_SPLIT):
    g = _geometry(case)
    exact = case["kind"] == "exact"
    dec = et.Executable(runtime(), batch=batch, max_tokens=max_tokens, block_size=BLOCK, kv_dtype=KV[kv][0], exact=exact,
                        max_advance=max_advance, rope_layout=rope, **g)
    ones = torch.ones(g["d_model"], device="cuda")
    embedding = torch.randn((g["vocab"], g["d_model"]), generator=gen, device="cuda").mul_(0.02)
    torch.cuda.synchronize()
    dec.set_weight(et.W_TOK_EMBD, 0, embedding)
    for layer in range(g["layers"]):
        dec.set_weight(et.W_ATTN_NORM, layer, ones)
        dec.set_weight(et.W_FFN_NORM, layer, ones)
    dec.set_weight(et.W_OUT_NORM, 0, ones)
    for slot, layer, rows, columns, codec in _projections(case):
        if codec == "f32":
            w = torch.randn((rows, columns), generator=gen, device="cuda").mul_(0.02)
            torch.cuda.synchronize()
            dec.set_weight(slot, layer, w)
        else:
            dec.set_weight(slot, layer, _packed(gen, codec, rows, columns), codec=CODECS[codec], rows=rows, columns=columns)
    dec.finalize()
    pool = et.NativeKvPool(runtime(), g["layers"], g["kv_heads"], g["head_dim"], max_tokens, BLOCK, KV[kv][0])
    return dec, pool, g


def _contexts(case):
    """Cached tokens of each lane, whole pages: the stated context, or spread from an eighth of it up to it."""
    pages = case["context"] // BLOCK
    if not case["ragged"]:
        return [case["context"]] * case["batch"]
    spread = np.random.default_rng(case["batch"] * 131 + pages).integers(max(1, pages // 8), pages + 1, size=case["batch"])
    return [int(p) * BLOCK for p in spread]


def _attention_lengths(case):
    rng = np.random.default_rng(case["batch"] * 8209 + case["longest"])
    return rng.integers(case["shortest"], case["longest"] + 1, size=case["batch"])


# ---------------------------------------------------------------------------------------------- prepare
def _prepare_decode(case, gen, rng):
    contexts, steps, batch = _contexts(case), case["steps"], case["batch"]
    max_tokens = sum(contexts) + batch * (steps // BLOCK + 3) * BLOCK
    dec, pool, g = _model(case, gen, batch, max_tokens, case["kv"], 1, ROPE[case["rope"]])
    # prompts of earlier requests fill the pages and stay in the prefix cache
    prompts = [rng.integers(0, g["vocab"], size=n + 1).astype(np.uint32) for n in contexts]
    earlier = [pool.makeSequence() for _ in contexts]
    for seq, prompt, n in zip(earlier, prompts, contexts):
        for layer in range(g["layers"]):
            k = torch.randn((1, g["kv_heads"], n, g["head_dim"]), generator=gen, device="cuda")
            v = torch.randn((1, g["kv_heads"], n, g["head_dim"]), generator=gen, device="cuda")
            torch.cuda.synchronize()
            runtime().kv_append_into(pool, layer, [seq], 1, 1, n, k, v, n)
        seq.commit(prompt[:n])
    for seq in earlier:
        seq.release()
    feed = rng.integers(0, g["vocab"], size=(steps, batch, 1)).astype(np.uint32)
    feed[0, :, 0] = [p[-1] for p in prompts]
    return dict(dec=dec, pool=pool, prompts=prompts, feed=feed)


def _prepare_prefill(case, gen, rng):
    batch, prompt = case["batch"], case["prompt"]
    max_tokens = batch * ((prompt + BLOCK - 1) // BLOCK + 2) * BLOCK
    dec, pool, g = _model(case, gen, batch, max_tokens, case["kv"], case["chunk"], ROPE[case["rope"]])
    return dict(dec=dec, pool=pool, tokens=rng.integers(0, g["vocab"], size=(batch, prompt)).astype(np.uint32))


def _prepare_exact(case, gen, rng):
    batch = case["batch"]
    max_tokens = batch * ((case["prompt"] + case["steps"] + BLOCK) // BLOCK + 1) * BLOCK
    dec, pool, g = _model(case, gen, batch, max_tokens, "f32", case["prompt"])
    return dict(dec=dec, pool=pool, tokens=rng.integers(0, g["vocab"], size=(batch, case["prompt"])).astype(np.uint32))


def _prepare_linear(case, gen, rng):
    rows, columns, vectors = case["rows"], case["columns"], case["vectors"]
    swiglu = case["epilogue"] == "swiglu"
    parts = [rows // 2] * 2 if swiglu else [rows]
    weights = [et.QWeight(runtime(), CODECS[case["weights"]], [_packed(gen, case["weights"], r, columns) for r in parts], parts, columns,
                          interleave8=swiglu) for _ in range(case["calls"])]
    out_columns = rows // 2 if swiglu else rows
    x = torch.randn((vectors, columns), generator=gen, device="cuda")
    residual = torch.randn((vectors, out_columns), generator=gen, device="cuda") if case["epilogue"] == "residual" else None
    outs = [torch.empty((vectors, out_columns), device="cuda") for _ in weights]
    size = weights[0].scratch_bytes(vectors)
    return dict(weights=weights, x=x, residual=residual, outs=outs, scratch=torch.empty(max(size, 4), dtype=torch.uint8, device="cuda"),
                scratch_bytes=size)


def _prepare_raw(case, gen, rng):
    x = torch.randn((case["vectors"], case["columns"]), generator=gen, device="cuda")
    return dict(x=x, packed=_packed(gen, case["weights"], case["rows"], case["columns"]),
                out=torch.empty((case["vectors"], case["rows"]), device="cuda"))


def _prepare_attention(case, gen, rng):
    rt = runtime()
    batch, kv_heads, head_dim, q_heads = case["batch"], case["kv_heads"], case["head_dim"], case["q_heads"]
    total = _attention_lengths(case)
    pages = sum(-(-int(n) // BLOCK) for n in total) + 1
    pool = et.NativeKvPool(rt, 1, kv_heads, head_dim, pages * BLOCK, BLOCK, KV[case["kv"]][0])
    seqs = [pool.makeSequence() for _ in range(batch)]
    grown = np.zeros(batch, dtype=np.int64)
    filler = np.zeros(BLOCK, dtype=np.uint32)
    while True:  # the sequences grow side by side, a page at a time and in changing order, so that their pages interleave
        left = np.minimum(total - grown, BLOCK)
        if not left.any():
            break
        for n in sorted({int(x) for x in left if x}):
            lanes = [int(i) for i in rng.permutation(np.flatnonzero(left == n))]
            k = torch.randn((len(lanes), kv_heads, n, head_dim), generator=gen, device="cuda")
            v = torch.randn((len(lanes), kv_heads, n, head_dim), generator=gen, device="cuda")
            torch.cuda.synchronize()
            rt.kv_append_into(pool, 0, [seqs[i] for i in lanes], len(lanes), len(lanes), n, k, v, n)
            for i in lanes:
                seqs[i].commit(filler[:n])
        grown += left
    lanes, table = np.zeros((batch, 4), dtype=np.int32), []
    for i, seq in enumerate(seqs):
        blocks, head = seq.blocks
        lanes[i] = (int(total[i]) - 1, 1, 0, len(table) - head)
        table.extend(int(b) for b in blocks)
    max_pages = -(-int(total.max()) // BLOCK)
    plan = et.attention_plan(batch, q_heads, kv_heads, head_dim, max_pages, sm_count=rt.capabilities()["sm_count"])
    return dict(pool=pool, seqs=seqs, lanes=torch.from_numpy(lanes).cuda(), tables=torch.tensor(table, dtype=torch.int32, device="cuda"),
                batch=batch, max_pages=max_pages, q=torch.randn((batch, q_heads, head_dim), generator=gen, device="cuda"), q_heads=q_heads,
                scale=1.0 / math.sqrt(head_dim), out=torch.empty((batch, q_heads, head_dim), device="cuda"),
                scratch=torch.empty(max(plan["partial_bytes"], 4), dtype=torch.uint8, device="cuda"), scratch_bytes=plan["partial_bytes"])


def _prepare_sample(case, gen, rng):
    rows = case["rows"]
    return dict(logits=torch.randn((rows, case["vocab"]), generator=gen, device="cuda").mul_(3.0), tokens=torch.empty(rows, dtype=torch.int32, device="cuda"),
                seeds=torch.from_numpy(rng.integers(0, 1 << 62, size=rows)).cuda(), counters=torch.from_numpy(rng.integers(0, 4096, size=rows)).cuda())


def _prepare_transcode(case, gen, rng):
    rows, columns, codec = case["rows"], case["columns"], case["weights"]
    state = dict(decoded=torch.empty((rows, columns), device="cuda"), x=None)
    if codec in K_SCALES:  # the library has no K-quant encoder: a file brings them packed
        state["packed"] = _packed(gen, codec, rows, columns)
    else:
        state["x"] = torch.randn((rows, columns), generator=gen, device="cuda").mul_(0.02)
        state["packed"] = torch.empty((rows, _row_bytes(codec, columns)), dtype=torch.uint8, device="cuda")
    return state


def prepare(case, seed):
    state = globals()["_prepare_" + case["kind"]](case, _generator(seed), np.random.default_rng(int(seed) + 1))
    state["case"] = case
    torch.cuda.synchronize()
    runtime().synchronize()
    return state


# ---------------------------------------------------------------------------------------------- run
def _run_decode(s):
    dec, pool = s["dec"], s["pool"]
    seqs = [pool.makeSequence() for _ in s["prompts"]]
    for seq, prompt in zip(seqs, s["prompts"]):
        seq.prefillMatch(prompt)
    step = dec.executeSampled if s["case"]["read"] == "tokens" else dec.execute
    out = [step(pool, seqs, tokens) for tokens in s["feed"]]
    for seq in seqs:
        seq.release()
    return out


def _run_prefill(s):
    dec, pool, tokens, chunk = s["dec"], s["pool"], s["tokens"], s["case"]["chunk"]
    seqs = [pool.makeSequence() for _ in range(tokens.shape[0])]
    first = 0
    while first + chunk < tokens.shape[1]:
        dec.executeSampled(pool, seqs, tokens[:, first:first + chunk])
        first += chunk
    logits = dec.execute(pool, seqs, tokens[:, first:])
    for seq in seqs:
        seq.release()
    return logits


def _run_exact(s):
    dec, pool, tokens = s["dec"], s["pool"], s["tokens"]
    seqs = [pool.makeSequence() for _ in range(tokens.shape[0])]
    logits = dec.execute(pool, seqs, tokens)
    generated, _ = dec.generate_greedy(pool, seqs, np.argmax(logits, axis=1), s["case"]["steps"])
    for seq in seqs:
        seq.release()
    return logits, generated


def _run_linear(s):
    epilogue = EPILOGUES[s["case"]["epilogue"]]
    for weight, out in zip(s["weights"], s["outs"]):
        weight.linear_into(s["x"], s["case"]["vectors"], out, residual=s["residual"], epilogue=epilogue, scratch=s["scratch"],
                           scratch_bytes=s["scratch_bytes"])
    return s["outs"]


def _run_raw(s):
    c = s["case"]
    runtime().qlinear_into(CODECS[c["weights"]], s["x"], c["vectors"], c["columns"], s["packed"], c["rows"], None, s["out"])
    return s["out"]


def _run_attention(s):
    runtime().paged_attention_into(s["pool"], 0, s["lanes"], s["tables"], s["batch"], s["max_pages"], s["q"], s["q_heads"], s["scale"],
                                   s["out"], s["scratch"], s["scratch_bytes"])
    return s["out"]


def _run_sample(s):
    c = s["case"]
    runtime().sample_rows_into(s["logits"], c["rows"], c["vocab"], s["tokens"], temperature=c["temperature"], top_k=c["top_k"] or None,
                               top_p=c["top_p"], seeds=s["seeds"], counters=s["counters"])
    return s["tokens"]


def _run_transcode(s):
    rt, c = runtime(), s["case"]
    if s["x"] is not None:
        rt.quantize_into(CODECS[c["weights"]], s["x"], c["rows"], c["columns"], s["packed"])
    rt.dequantize_into(CODECS[c["weights"]], s["packed"], c["rows"], c["columns"], s["decoded"])
    return s["packed"], s["decoded"]


def run(state):
    return globals()["_run_" + state["case"]["kind"]](state)


# ---------------------------------------------------------------------------------------------- work, tolerance
def _matrix_bytes(codec, rows, columns):
    return rows * columns * 4 if codec == "f32" else rows * _row_bytes(codec, columns)


def _step_work(case, lanes, tokens, cached, kv):
    """One invocation of a model on lanes x tokens rows whose lanes have `cached` tokens (a list) behind them."""
    g = _geometry(case)
    rows = lanes * tokens
    size = KV[kv][1] + (4.0 / g["head_dim"] if kv == "u8" else 0.0)
    row = 2 * g["layers"] * g["kv_heads"] * g["head_dim"] * size
    attended = sum(tokens * n + tokens * (tokens + 1) / 2 for n in cached)
    total = rows * g["d_model"] * 4 + row * (sum(cached) + 2 * rows)
    flops = 4.0 * attended * g["q_heads"] * g["head_dim"] * g["layers"]
    for slot, _, r, c, codec in _projections(case):
        total += _matrix_bytes(codec, r, c)
        flops += 2.0 * r * c * (lanes if slot == et.W_HEAD else rows)
    return total, flops


def work(case):
    kind = case["kind"]
    parts = []
    if kind == "decode":
        contexts = _contexts(case)
        out = case["batch"] * 4 * (1 if case["read"] == "tokens" else _geometry(case)["vocab"])
        parts = [_step_work(case, case["batch"], 1, [n + t for n in contexts], case["kv"]) for t in range(case["steps"])]
        parts.append((out * case["steps"], 0))
    elif kind == "prefill":
        for first in range(0, case["prompt"], case["chunk"]):
            n = min(case["chunk"], case["prompt"] - first)
            parts.append(_step_work(case, case["batch"], n, [first] * case["batch"], case["kv"]))
        parts.append((case["batch"] * 4 * _geometry(case)["vocab"], 0))
    elif kind == "exact":
        b = case["batch"]
        parts = [_step_work(case, b, case["prompt"], [0] * b, "f32")]
        parts += [_step_work(case, b, 1, [case["prompt"] + t] * b, "f32") for t in range(case["steps"])]
        parts.append((b * 4 * (case["vocab"] + case["steps"]), 0))
    elif kind in ("linear", "raw"):
        out_columns = case["rows"] // 2 if case.get("epilogue") == "swiglu" else case["rows"]
        io = case["vectors"] * 4 * (case["columns"] + out_columns * (2 if case.get("epilogue") == "residual" else 1))
        calls = case.get("calls", 1)
        parts = [(calls * (_matrix_bytes(case["weights"], case["rows"], case["columns"]) + io), calls * 2.0 * case["vectors"] * case["rows"] * case["columns"])]
    elif kind == "attention":
        total = int(_attention_lengths(case).sum())
        size = KV[case["kv"]][1] + (4.0 / case["head_dim"] if case["kv"] == "u8" else 0.0)
        parts = [(total * 2 * case["kv_heads"] * case["head_dim"] * size + case["batch"] * case["q_heads"] * case["head_dim"] * 8,
                  4.0 * total * case["q_heads"] * case["head_dim"])]
    elif kind == "sample":
        parts = [(case["rows"] * (case["vocab"] * 4 + 20), 2.0 * case["rows"] * case["vocab"])]
    else:
        packed, plain = _matrix_bytes(case["weights"], case["rows"], case["columns"]), case["rows"] * case["columns"] * 4
        coded = case["weights"] not in K_SCALES
        parts = [((plain + packed if coded else 0) + packed + plain, (4.0 if coded else 2.0) * case["rows"] * case["columns"])]
    return {"bytes": float(sum(p[0] for p in parts)), "flops": float(sum(p[1] for p in parts))}


def tolerance(case):
    kind = case["kind"]
    if kind in ("decode", "prefill"):
        # f16 (or bf16) operands in every projection and in attention, layer after layer; "differ": near-ties of the argmax
        return {"rel": 2e-2 if case["kv"] == "bf16" else 1e-2, "differ": 0.01}
    if kind == "exact":
        return {"rel": 1e-5, "differ": 0.01}
    if kind in ("linear", "attention"):
        return {"rel": 1e-2 if case.get("kv") == "bf16" else 2e-3}
    if kind == "raw":
        return {"rel": 1e-5}  # f32 sums of exactly decoded weights
    return "exact"  # token ids, packed bytes, decoded values
