"""Performance cases of the engine: the calls that a program running 4-bit / 8-bit models makes.

Four kinds of work, all through the Python binding of the C ABI:

  gemm      Context.gemv_q4 / gemm_q4 over a packed weight (4-bit, 8-bit or K-quant blocks), from one
            activation row (decoding) over a decode batch and a prompt chunk to thousands of rows
            (prompt phase), with f32, bf16 or f16 activations and odd row counts and widths
  attn      Context.attn_decode over a paged f16 KV cache: one long conversation, or a ragged batch;
            soft-capped and windowed forms as some model families use them
  generate  the layer executor: a request as the mind loop serves it (prompt in chunks with progress,
            then one decode call per streamed token), a batch of sequences decoded together, and a long
            prompt taken in one call; the 32-layer, 4096-wide decoder of the benchmark

Weights, the KV cache, the decoder and the context are what a program holds while it serves calls, so
`prepare` makes them (the decoder once per process: a server loads its model once and its requests
differ in their prompts); `run` makes the calls.
"""
import math

import numpy as np
import torch

from cyb_b200 import qeng

DT = {"f32": torch.float32, "bf16": torch.bfloat16, "f16": torch.float16}
BLOCK_BYTES = {"q4": 0.5625, "q8": 1.0625, "q4k": 0.5625}  # per weight

# the decoder of the benchmark: 7B-shaped, 4-bit blocks
MODEL = dict(layers=32, d_model=4096, ffn=11008, heads=32, kv_heads=8, vocab=32000)
MAX_BATCH, MAX_SEQ = 16, 2304

_ctx = None
_decoder = None


def context():
    global _ctx
    if _ctx is None:
        _ctx = qeng.Context(0)
    return _ctx


def listed():
    return [
        # one token through one attention-sized projection: the smallest call, latency and host path
        {"name": "gemv-4096", "kind": "gemm", "fmt": "q4", "m": 1, "n": 4096, "k": 4096, "x": "f32"},
        # one token through the fused gate|up matrix of an 8-bit model: the bandwidth case
        {"name": "gemv-q8-gateup", "kind": "gemm", "fmt": "q8", "m": 1, "n": 22016, "k": 4096, "x": "f32"},
        # a decode batch of 8 sequences, gate or up projection
        {"name": "batch8-up", "kind": "gemm", "fmt": "q4", "m": 8, "n": 11008, "k": 4096, "x": "bf16"},
        # a decode batch of 32 sequences, down projection
        {"name": "batch32-down", "kind": "gemm", "fmt": "q4", "m": 32, "n": 4096, "k": 11008, "x": "bf16"},
        # a short prompt or the remainder of a chunked one (an odd row count, f32 rows as the executor has them)
        {"name": "chunk101-up", "kind": "gemm", "fmt": "q4", "m": 101, "n": 11008, "k": 4096, "x": "f32"},
        # a medium prompt whose length fits no tile
        {"name": "prefill777-up", "kind": "gemm", "fmt": "q4", "m": 777, "n": 11008, "k": 4096, "x": "f32"},
        # many prompts at once, down projection: the largest contraction
        {"name": "prefill8192-down", "kind": "gemm", "fmt": "q4", "m": 8192, "n": 4096, "k": 11008, "x": "bf16"},
        # decode attention of a serving batch with ragged contexts
        {"name": "attn-batch16", "kind": "attn", "batch": 16, "lo": 512, "hi": 4096, "heads": 32, "kv_heads": 8,
         "softcap": 0.0, "window": 0},
        # decode attention of one long conversation
        {"name": "attn-long", "kind": "attn", "batch": 1, "lo": 15001, "hi": 15001, "heads": 32, "kv_heads": 8,
         "softcap": 0.0, "window": 0},
        # a question with its recalled context: the prompt in chunks of 128 (progress events), then one
        # decode call per streamed token
        {"name": "ask", "kind": "generate", "batch": 1, "prompt": 300, "chunk": 128, "new": 48, "stream": True},
        # sixteen sequences decoded together
        {"name": "serve16", "kind": "generate", "batch": 16, "prompt": 45, "chunk": 0, "new": 24, "stream": False},
        # a document read in one call, first token out
        {"name": "prompt1800", "kind": "generate", "batch": 1, "prompt": 1800, "chunk": 0, "new": 1, "stream": False},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["gemm", "gemm", "gemm", "gemm", "attn", "attn", "generate"])
    if kind == "gemm":
        fmt = rng.choice(["q4", "q4", "q4", "q8", "q4k"])
        big = rng.random() < 0.7
        if fmt == "q4k":  # super-blocks of 256 along K
            n, k = rng.choice([(4096, 4096), (11008, 4096)]) if big else (16 * _log(rng, 32, 700), 256 * rng.randint(2, 20))
        else:
            n, k = (rng.choice([(4096, 4096), (6144, 4096), (11008, 4096), (22016, 4096), (4096, 11008)]) if big
                    else (16 * _log(rng, 32, 1400), 32 * _log(rng, 16, 350)))
        # prompts of 8-bit and K-quant models come in chunks; 4-bit prompts up to thousands of rows
        m = _log(rng, 1, 8192 if fmt == "q4" else 256)
        x = rng.choice(["f32", "bf16"]) if m >= 256 else rng.choice(["f32", "bf16", "f16"])
        return {"kind": "gemm", "fmt": fmt, "m": m, "n": n, "k": k, "x": x}
    if kind == "attn":
        b = _log(rng, 1, 24)
        hi = _log(rng, 64, min(20000, 65536 // b))
        heads, kv = rng.choice([(32, 8), (32, 8), (16, 8), (32, 32), (64, 8), (12, 2)])
        return {"kind": "attn", "batch": b, "lo": max(1, hi // 8), "hi": hi, "heads": heads, "kv_heads": kv,
                "softcap": rng.choice([0.0, 0.0, 0.0, 30.0]), "window": rng.choice([0, 0, 0, 1024])}
    b = rng.choice([1, 1, 1, 2, 3, 4, 7, 8, 12, 16])
    prompt = _log(rng, 8, 1800 // b)
    stream = b == 1 and rng.random() < 0.5
    return {"kind": "generate", "batch": b, "prompt": prompt, "chunk": 128 if stream else 0,
            "new": _log(rng, 2, 48 if b == 1 else 16), "stream": stream}


# ---- states -----------------------------------------------------------------------------------
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _weight(case, seed):
    n, k, fmt, ctx = case["n"], case["k"], case["fmt"], context()
    if fmt == "q4k":
        # super-blocks of 144 bytes: f16 d and dmin, 12 bytes of 6-bit scales and minima, 128 bytes of codes
        rng = np.random.Generator(np.random.PCG64(seed))
        blocks = rng.integers(0, 256, (n * k // 256, 144), dtype=np.uint8)
        d = rng.uniform(2e-4, 6e-4, (n * k // 256, 2)).astype(np.float16)
        blocks[:, :4] = d.view(np.uint8)
        return ctx.pack_q4k(blocks, n, k)
    w = torch.randn(n, k, device="cuda", generator=_gen(seed)) * 0.05
    return ctx.quantize_q4(w) if fmt == "q4" else ctx.quantize_q8(w)


def _prepare_gemm(case, seed):
    w = _weight(case, seed)
    x = torch.randn(case["m"], case["k"], device="cuda", generator=_gen(seed + 1)).to(DT[case["x"]])
    return {"kind": "gemm", "ctx": context(), "w": w, "x": x, "row": x[0] if case["m"] == 1 and case["x"] == "f32" else None}


def _prepare_attn(case, seed):
    ctx = context()
    rng = np.random.Generator(np.random.PCG64(seed))
    b, hkv = case["batch"], case["kv_heads"]
    lens = rng.integers(case["lo"], case["hi"] + 1, b).astype(np.int32)
    npages = (lens + 15) // 16
    total = int(npages.sum())
    pool = ctx.kv_pool(total, hkv)
    pool.tensor().normal_(generator=_gen(seed))
    order = rng.permutation(total).astype(np.int32)
    # the table has room for the longest context the cache admits
    table = np.zeros((b, (case["hi"] + 15) // 16), np.int32)
    off = 0
    for i in range(b):
        table[i, :npages[i]] = order[off:off + npages[i]]
        off += npages[i]
    q = torch.randn(b, case["heads"], 128, device="cuda", generator=_gen(seed + 1)).half()
    return {"kind": "attn", "ctx": ctx, "pool": pool, "q": q, "table": torch.from_numpy(table).cuda(),
            "lens": torch.from_numpy(lens).cuda(), "softcap": case["softcap"], "window": case["window"]}


def decoder():
    """The served model, loaded once per process.  Its weights are random 4-bit blocks; the head is the
    embedding table in another row order, so that the next token stands out as it does in a trained model
    (independent random tables leave near-ties, which any change of summation order would resolve
    differently), while every logit still depends on what the layers add to the residual stream."""
    global _decoder
    if _decoder is not None:
        return _decoder
    c = MODEL
    dec = context().decoder(max_batch=MAX_BATCH, max_seq=MAX_SEQ, **c)
    d, f, hd = c["d_model"], c["ffn"], 128
    nq, nkv = c["heads"] * hd, c["kv_heads"] * hd
    shapes = [(nq, d), (nkv, d), (nkv, d), (d, nq), (f, d), (f, d), (d, f)]
    g = _gen(1)
    mats = []
    for n, k in shapes:  # every layer gets these numbers: only the time to make them is saved
        q = torch.randint(0, 16, (n, k), device="cuda", generator=g, dtype=torch.uint8).cpu().numpy()
        s = (torch.rand(n, k // 32, device="cuda", generator=g) * 0.0018 + 0.0002).half().cpu().numpy()
        mats.append((q, s))
    ones = np.ones(d, np.float32)
    for layer in range(c["layers"]):
        for which, (q, s) in enumerate(mats):
            dec.load_matrix(layer, which, q, s)
        dec.load_norm(layer, 0, ones)
        dec.load_norm(layer, 1, ones)
    emb = torch.randn(c["vocab"], d, device="cuda", generator=g)
    perm = torch.randperm(c["vocab"], device="cuda", generator=g)
    bits = lambda t: t.bfloat16().view(torch.int16).cpu().numpy().view(np.uint16)  # noqa: E731
    dec.load_head(bits(emb), bits(emb[perm] * 0.02), ones)
    _decoder = dec
    return dec


def _prepare_generate(case, seed):
    rng = np.random.Generator(np.random.PCG64(seed))
    prompt = rng.integers(0, MODEL["vocab"], (case["batch"], case["prompt"])).astype(np.int32)
    return {"kind": "generate", "dec": decoder(), "prompt": prompt, "chunk": case["chunk"], "new": case["new"], "stream": case["stream"]}


def prepare(case, seed):
    return {"gemm": _prepare_gemm, "attn": _prepare_attn, "generate": _prepare_generate}[case["kind"]](case, seed)


# ---- one pass ---------------------------------------------------------------------------------
def run(state):
    if state["kind"] == "gemm":
        if state["row"] is not None:
            return state["ctx"].gemv_q4(state["w"], state["row"])
        return state["ctx"].gemm_q4(state["w"], state["x"])
    if state["kind"] == "attn":
        return state["ctx"].attn_decode(state["pool"], state["q"], state["table"], state["lens"],
                                        softcap=state["softcap"], window=state["window"])
    dec, prompt = state["dec"], state["prompt"]
    dec.reset(prompt.shape[0])
    step = state["chunk"] or prompt.shape[1]
    for p in range(0, prompt.shape[1], step):
        dec.prefill(prompt[:, p:p + step])
    if state["stream"]:
        tokens = np.concatenate([dec.decode(1) for _ in range(state["new"])], 1)
    else:
        tokens = dec.decode(state["new"])
    # the next token's distribution comes along (log-probabilities, host-side sampling)
    return {"tokens": tokens, "logits": dec.logits()}


# ---- what a pass cannot do without --------------------------------------------------------------
def work(case):
    if case["kind"] == "gemm":
        m, n, k = case["m"], case["n"], case["k"]
        esz = 4 if case["x"] == "f32" else 2
        return {"bytes": n * k * BLOCK_BYTES[case["fmt"]] + m * k * esz + m * n * 4, "flops": 2.0 * m * n * k}
    if case["kind"] == "attn":
        tokens = case["batch"] * (case["lo"] + case["hi"]) / 2.0
        if case["window"]:
            tokens = min(tokens, case["batch"] * float(case["window"]))
        return {"bytes": tokens * case["kv_heads"] * 2 * 128 * 2 + case["batch"] * case["heads"] * 128 * 6,
                "flops": 4.0 * tokens * case["heads"] * 128}
    c = MODEL
    b, p, new = case["batch"], case["prompt"], case["new"]
    nq, nkv = c["heads"] * 128, c["kv_heads"] * 128
    weights = c["layers"] * (c["d_model"] * (2 * nq + 2 * nkv) + 3 * c["d_model"] * c["ffn"])
    head = c["vocab"] * c["d_model"]
    calls = -(-p // case["chunk"]) if case["chunk"] else 1
    kv_token = c["layers"] * nkv * 2 * 2  # bytes of one token's keys and values
    kv = b * kv_token * (p + sum(p + i + 1 for i in range(new)))
    flops = 2.0 * b * (p + new) * weights + 2.0 * b * (new + 1) * head
    flops += 4.0 * b * c["layers"] * nq * (p * (p + 1) / 2.0 + sum(p + i + 1 for i in range(new)))
    return {"bytes": (calls + new) * weights * BLOCK_BYTES["q4"] + (new + 1) * head * 2.0 + kv, "flops": flops}


def tolerance(case):
    if case["kind"] == "gemm":
        if case["m"] >= 256 and case["fmt"] == "q4":
            return {"rel": 5e-3, "max": 0.05}  # prompt path: operands rounded to bf16
        if case["m"] == 1:
            return {"rel": 1e-5, "max": 1e-4}  # activations in 22 bits, 32-bit sums
        return {"rel": 3e-4, "max": 3e-3}      # activations in 15 bits per block
    if case["kind"] == "attn":
        return {"rel": 1e-4, "max": 2e-3}      # f16 operands, 32-bit softmax and sums
    # 32 layers with bf16 prompt operands and 15-bit decode activations
    return {"rel": 1e-2, "max": 0.2, "differ": 0.01}
