"""Matmuls of several rows (bf16 operands in two terms, tensor-memory and mma.sync kernels) and the prompt path at the
edges of their tiles, against float64 arithmetic."""
import numpy as np
import pytest

from oracle import ref

pytestmark = pytest.mark.gpu
DT = ("float32", "bfloat16", "float16")


def _weight(ctx, fmt, n, k):
    import torch
    g = torch.Generator(device="cuda")
    g.manual_seed(7)
    if fmt == "q4k":
        _, _, blocks = ref.make_q4k(ref.rng_of(7), n, k)
        return ctx.pack_q4k(blocks, n, k)
    w = torch.randn(n, k, device="cuda", generator=g) * 0.05
    return ctx.quantize_q4(w) if fmt == "q4" else ctx.quantize_q8(w)


# Rows: the smallest and largest of the mma.sync kernel's column tiles, of the tensor-memory kernel's token tiles (16 to
# 256) and of its two- and one-chunk stages.  N: one row tile, a remainder of 256; K: one block, an odd block count, one
# that cuts tiles along K.
# Bound: an operand in two bf16 terms is off by 2^-17 of itself at most, bf16 operands by nothing; f32 sums of K products
# in chains of up to K / 16 tensor-core steps that truncate add K / 16 * 2^-24 of the running sum: 3e-5 covers both at
# these K (the random errors measured are ten times smaller).
@pytest.mark.parametrize("fmt", ["q4", "q8", "q4k"])
@pytest.mark.parametrize("m", [3, 5, 8, 9, 16, 17, 32, 33, 64, 65, 112, 113, 129, 255])
def test_rows_and_widths(ctx, fmt, m):
    import torch
    shapes = [(16, 256), (272, 768)] if fmt == "q4k" else [(16, 32), (272, 736), (1040, 992)]
    for i, (n, k) in enumerate(shapes):
        w = _weight(ctx, fmt, n, k)
        wd = w.dequant().double()
        for dt in DT:
            if dt != "bfloat16" and m < 5:
                continue  # those rows take the integer kernel (tests of its own)
            x = torch.randn(m, k, device="cuda").to(getattr(torch, dt))
            y = torch.full((m, n + 8), 0.25, device="cuda")[:, :n]
            acc = (m + i) % 2
            ctx.gemm_q4(w, x, out=y, flags=acc)
            want = x.double() @ wd.T + (0.25 if acc else 0.0)
            err = float((y.double() - want).abs().max() / want.abs().max())
            assert err < 3e-5, (fmt, m, n, k, dt, err)
    ctx.device_status()


# Rows that the matmul converts itself: odd row starts and strides (no 16-byte loads), f16, bf16 rows that are not aligned, slices of
# which the last is short, rows that fill no column tile.  Bound as above.
@pytest.mark.parametrize("fmt", ["q4", "q8", "q4k"])
@pytest.mark.parametrize("m,n,k,off,pad", [(5, 272, 768, 1, 0), (16, 1040, 4352, 3, 5), (7, 2064, 2304, 0, 1), (11, 48, 11008, 2, 0)])
def test_few_rows_of_any_alignment(ctx, fmt, m, n, k, off, pad):
    import torch
    w = _weight(ctx, fmt, n, k)
    wd = w.dequant().double()
    for dt in DT:
        x = torch.randn(off + m * (k + pad), device="cuda").to(getattr(torch, dt))[off:].view(m, k + pad)[:, :k]
        want = x.double() @ wd.T
        assert float((ctx.gemm_q4(w, x).double() - want).abs().max() / want.abs().max()) < 3e-5, (fmt, m, n, k, dt)
    ctx.device_status()


# Three and four f32 / f16 rows around the line from which tall matrices leave the integer kernel (whose 15-bit activations give
# 2e-4): 40000 values of activations, K above N.  Above it the bound of the planes.  Which kernel it was shows where one value of
# every block of 32 (its weights are zero) is 2^16 times the largest of the others: nothing is left of those in fixed point per block.
@pytest.mark.parametrize("fmt", ["q4", "q8"])
@pytest.mark.parametrize("m,n,k,planes", [(4, 4096, 10016, True), (4, 272, 9984, False), (3, 1040, 13344, True), (4, 10016, 10016, False)])
def test_few_rows_of_tall_matrices(ctx, fmt, m, n, k, planes):
    import torch
    w = torch.randn(n, k, device="cuda") * 0.05
    w[:, ::32] = 0.0
    w = ctx.quantize_q4(w) if fmt == "q4" else ctx.quantize_q8(w)
    wd = w.dequant().double()
    for dt in ("float32", "float16"):
        x = torch.randn(m, k, device="cuda").to(getattr(torch, dt))
        want = x.double() @ wd.T
        err = float((ctx.gemm_q4(w, x).double() - want).abs().max() / want.abs().max())
        assert err < (3e-5 if planes else 2e-4), (fmt, m, n, k, dt, err)
        x = (torch.rand(m, k, device="cuda") * 2.0 ** -16).to(getattr(torch, dt))
        x[:, ::32] = 1.0
        want, y = x.double() @ wd.T, ctx.gemm_q4(w, x).double()
        if planes:
            assert float((y - want).abs().max() / want.abs().max()) < 3e-5, (fmt, m, n, k, dt)
        else:
            assert not bool(y.any()), (fmt, m, n, k, dt)
    ctx.device_status()


# Four sequences whose down projection is tall enough for the batch kernel take it for the whole layer.  Against the teacher; an
# operand of 17 bits keeps far below 2e-3.
def test_four_sequences_with_a_tall_down_projection(ctx):
    from cyb_b200 import qeng
    cfg = ref.DecoderConfig(layers=2, d=256, ffn=10240, heads=4, kv_heads=2, vocab=320)
    W = ref.make_decoder_weights(cfg, seed=8)
    dec = ctx.decoder(layers=2, d_model=256, ffn=10240, heads=4, kv_heads=2, vocab=320, max_batch=4, max_seq=32)
    qeng.load_decoder_weights(dec, W, cfg)
    prompt = ref.rng_of(4).integers(0, 320, (4, 3)).astype(np.int32)
    dec.reset(4)
    dec.prefill(prompt)
    want, logs = ref.Decoder(cfg, W).generate(prompt, 6)
    assert ref.err_inf(dec.logits(), logs[0]) < 2e-3
    toks = dec.decode(6)
    # a token may differ only where the teacher's two best logits are closer than the gate; what follows it is then free
    for b in range(4):
        for s in range(6):
            if toks[b, s] != want[b, s]:
                top = np.sort(logs[s][b])[-2:]
                assert top[1] - top[0] < 2e-3 * np.abs(logs[s][b]).max(), (b, s)
                break
    ctx.device_status()
    dec.free()


def _plan(ctx, w, m, wp, xp, epilogue):
    """What the planner of the many-row matmul chose, for the tests below to know what they ran."""
    import ctypes
    from cyb_b200 import qeng
    out = (ctypes.c_int32 * 6)()
    fn = qeng._lib.qeng_many_rows_plan
    fn.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_int64, ctypes.c_int32, ctypes.c_int32, ctypes.c_int32, ctypes.c_void_p]
    assert fn(ctx.h, w.h, m, wp, xp, epilogue, out) == 0
    chunks, width, accumulators, whole, cut, pairs = out
    kind = "mixed" if whole and cut else "cut" if cut else "rounds" if whole > pairs else "one round"
    return chunks, width, accumulators, kind


# Every kind of plan: stages of two chunks or one, one accumulator (which the dequantising warps help to add to y) or two,
# tiles all whole (one round, or several to a pair), all cut along K, or both; rows and widths that fill no tile; the widest
# tile.  Stored and added to y.  One weight term (256 rows of 4-bit blocks and more) against operands rounded to bf16, two
# against exact ones; bound as above.
@pytest.mark.parametrize("fmt,m,n,k,plan", [
    ("q4", 412, 7360, 288, (2, 208, 1, "one round")), ("q4", 649, 12432, 544, (2, 224, 1, "rounds")),
    ("q4", 823, 1840, 5792, (2, 208, 1, "cut")), ("q4", 321, 10720, 5504, (2, 176, 1, "mixed")),
    ("q4", 260, 19792, 544, (2, 144, 2, "rounds")), ("q4", 271, 272, 3488, (2, 80, 2, "cut")),
    ("q4", 260, 9504, 5248, (2, 96, 2, "mixed")), ("q4", 2025, 4112, 4096, (2, 256, 1, "rounds")),
    ("q4", 206, 10288, 320, (1, 208, 1, "one round")), ("q8", 167, 18960, 1408, (1, 176, 1, "rounds")),
    ("q8", 197, 5424, 3616, (1, 208, 1, "cut")), ("q8", 194, 20864, 1664, (1, 208, 1, "mixed")),
    ("q4", 207, 19232, 256, (1, 112, 2, "rounds")), ("q4", 161, 304, 3488, (1, 80, 2, "cut")),
    ("q8", 33, 20640, 2144, (1, 48, 2, "mixed")), ("q8", 73, 448, 480, (2, 80, 1, "one round")),
    ("q4", 78, 19776, 864, (2, 80, 1, "rounds")), ("q8", 65, 10400, 3168, (2, 80, 1, "cut")),
    ("q4", 67, 20512, 2816, (2, 80, 1, "mixed")), ("q4", 33, 336, 1984, (2, 48, 2, "cut")),
    ("q8", 38, 21712, 1920, (2, 48, 2, "mixed"))])
def test_every_kind_of_plan(ctx, fmt, m, n, k, plan):
    import torch
    w = _weight(ctx, fmt, n, k)
    one_term = fmt == "q4" and m >= 256
    rounded = (lambda t: t.bfloat16()) if one_term else (lambda t: t)
    wd = rounded(w.dequant()).double()
    for acc in (0, 1):
        assert _plan(ctx, w, m, 1 if one_term else 2, 1 if one_term else 2, acc) == plan
        for dt in DT[:2] if one_term else DT[:1]:
            x = torch.randn(m, k, device="cuda").to(getattr(torch, dt))
            y = torch.full((m + 1, n + 8), 0.25, device="cuda")
            ctx.gemm_q4(w, x, out=y[:m, :n], flags=acc)
            want = rounded(x).double() @ wd.T + (0.25 if acc else 0.0)
            err = float((y[:m, :n].double() - want).abs().max() / want.abs().max())
            assert err < 3e-5, (fmt, m, n, k, acc, dt, err)
            assert bool((y[m] == 0.25).all()) and bool((y[:, n:] == 0.25).all())
    ctx.device_status()


# Layers narrower than 2048: 4-bit blocks (one term), several tiles a pair through two accumulators; 8-bit (two), several through
# one, then cut ones.
@pytest.mark.parametrize("fmt,d,plan", [("q4", 512, (2, "rounds")), ("q8", 256, (1, "mixed"))])
def test_prompt_epilogues_over_several_tiles(ctx, fmt, d, plan):
    """Rotary embedding with KV append, SwiGLU and the residual adds where CTA pairs run several tiles: a layer over 895 rows against
    the float64 teacher (operands rounded to bf16: 5e-3)."""
    import torch
    from cyb_b200 import qeng
    T = 895
    cfg = ref.DecoderConfig(layers=1, d=d, ffn=4096, heads=32, kv_heads=8, vocab=320)
    W = ref.make_decoder_weights(cfg, seed=5, fmt=fmt)
    dec = ctx.decoder(layers=1, d_model=d, ffn=4096, heads=32, kv_heads=8, vocab=320, max_batch=1, max_seq=896)
    qeng.load_decoder_weights(dec, W, cfg)
    SWIGLU, QKV = 3, 4
    terms = 1 if fmt == "q4" else 2
    assert _plan(ctx, dec.weight(0, 0), T, terms, terms, QKV)[2:] == plan
    assert _plan(ctx, dec.weight(0, 2), T, terms, terms, SWIGLU)[2:] == plan
    teacher = ref.Decoder(cfg, W)
    teacher.reset(1)
    x = ref.rng_of(41).standard_normal((1, T, cfg.d), dtype=np.float32)
    want = teacher.layer(0, x.astype(np.float64), np.arange(T)[None])
    got = dec.layer(0, torch.from_numpy(x[0]).cuda(), np.arange(T)).cpu().numpy()
    ctx.device_status()
    assert ref.err_inf(got, want[0]) < 5e-3
    dec.free()


def test_prompt_epilogues_of_whole_tiles(ctx):
    """The same over a wider matrix (K of 2048), with whole tiles of more tokens than a multiple of 16.  Against the teacher the
    operands rounded to bf16 leave 1e-2 here (the second matrix sees products of two of them); against the same rows in two calls,
    in other tiles, only the roundings tipped by sums in another order differ (2^-9 of single operands: 1e-3).  Three sequences
    give the same in another order."""
    import torch
    from cyb_b200 import qeng
    T = 601
    cfg = ref.DecoderConfig(layers=1, d=2048, ffn=4096, heads=16, kv_heads=8, vocab=320)
    W = ref.make_decoder_weights(cfg, seed=5)
    dec = ctx.decoder(layers=1, d_model=2048, ffn=4096, heads=16, kv_heads=8, vocab=320, max_batch=3, max_seq=640)
    qeng.load_decoder_weights(dec, W, cfg)
    SWIGLU, QKV = 3, 4
    for rows in (T, 3 * 173):
        assert _plan(ctx, dec.weight(0, 0), rows, 1, 1, QKV)[3] != "cut" and _plan(ctx, dec.weight(0, 2), rows, 1, 1, SWIGLU)[3] != "cut"
    teacher = ref.Decoder(cfg, W)
    teacher.reset(1)
    x = ref.rng_of(41).standard_normal((1, T, cfg.d), dtype=np.float32)
    want = teacher.layer(0, x.astype(np.float64), np.arange(T)[None])
    xs = torch.from_numpy(x[0]).cuda()
    got = dec.layer(0, xs, np.arange(T)).cpu().numpy()
    assert ref.err_inf(got, want[0]) < 2e-2
    halves = [dec.layer(0, xs[a:b], np.arange(a, b)).cpu().numpy() for a, b in ((0, 301), (301, T))]
    assert ref.err_inf(np.concatenate(halves), got) < 4e-3
    prompt = ref.rng_of(43).integers(0, 320, (3, 173)).astype(np.int32)
    logits = []
    for order in ([0, 1, 2], [2, 0, 1]):
        dec.reset(3)
        dec.prefill(prompt[order])
        logits.append(dec.logits()[np.argsort(order)])
    assert ref.err_inf(logits[1], logits[0]) < 1e-3
    ctx.device_status()
    dec.free()


# Query heads per kv head: one, the most there are, and counts that do not divide the 128 rows of a prompt attention tile
# (its last rows stay empty); tiles then hold 128, 16, 42, 25, 21 and 18 tokens.
@pytest.mark.parametrize("heads,kv_heads", [(2, 2), (8, 1), (6, 2), (5, 1), (6, 1), (7, 1)])
def test_prompt_attention_groups(ctx, heads, kv_heads):
    from cyb_b200 import qeng
    cfg = ref.DecoderConfig(layers=2, d=256, ffn=512, heads=heads, kv_heads=kv_heads, vocab=320)
    W = ref.make_decoder_weights(cfg, seed=5)
    dec = ctx.decoder(layers=2, d_model=256, ffn=512, heads=heads, kv_heads=kv_heads, vocab=320, max_batch=2, max_seq=128)
    qeng.load_decoder_weights(dec, W, cfg)
    prompt = ref.rng_of(heads).integers(0, 320, (2, 86)).astype(np.int32)
    dec.reset(2)
    dec.prefill(prompt[:, :65])
    dec.prefill(prompt[:, 65:])
    want, logs = ref.Decoder(cfg, W).generate(prompt, 3)
    assert ref.err_inf(dec.logits(), logs[0]) < 2e-3
    assert np.array_equal(dec.decode(3), want)
    ctx.device_status()
    dec.free()


# Norms of prompt rows wider than what a thread block keeps in registers (4096 values from two rows to an SM on, 8192 below): the rest
# is read twice, here one warp's loads, or two blocks of 1024 with a remainder.  Operands of 17 bits (8-bit blocks, or fewer than 256
# rows), so rounding stays far below 2e-3.
@pytest.mark.parametrize("d,rows,fmt", [(4224, 300, "q8"), (6528, 300, "q8"), (8256, 20, "q4")])
def test_norm_of_wide_prompt_rows(ctx, d, rows, fmt):
    from cyb_b200 import qeng
    cfg = ref.DecoderConfig(layers=1, d=d, ffn=512, heads=2, kv_heads=1, vocab=320)
    W = ref.make_decoder_weights(cfg, seed=7, fmt=fmt)
    dec = ctx.decoder(layers=1, d_model=d, ffn=512, heads=2, kv_heads=1, vocab=320, max_batch=1, max_seq=304)
    qeng.load_decoder_weights(dec, W, cfg)
    prompt = ref.rng_of(d).integers(0, 320, (1, rows)).astype(np.int32)
    dec.reset(1)
    dec.prefill(prompt)
    _, logs = ref.Decoder(cfg, W).generate(prompt, 1)
    assert ref.err_inf(dec.logits(), logs[0]) < 2e-3
    ctx.device_status()
    dec.free()


# More tiles of the prompt attention than SMs: two to a CTA, an odd number of them, ten tiles of keys through a ring of three, and
# scores spread so far that rows are rescaled on the way.  Against the teacher the operands of the matmuls, rounded to bf16 (2^-9
# each, of scores of some tens), leave 1e-2 (as much with any attention); against the same prompt in two calls, one tile a CTA,
# only sums in another order differ, and the bf16 roundings of its output that they tip: far below 1e-3.
@pytest.mark.parametrize("window", [0, 100])
def test_long_prompt_attention_two_tiles_a_cta(ctx, window):
    import torch
    from cyb_b200 import qeng
    cfg = ref.DecoderConfig(layers=1, d=256, ffn=512, heads=8, kv_heads=1, vocab=320, sliding_window=window)
    W = ref.make_decoder_weights(cfg, seed=6)
    q, s = W["layers"][0]["wq"]
    W["layers"][0]["wq"] = (q, (s.astype(np.float32) * 4).astype(np.float16))
    dec = ctx.decoder(layers=1, d_model=256, ffn=512, heads=8, kv_heads=1, vocab=320, max_batch=4, max_seq=640, sliding_window=window)
    qeng.load_decoder_weights(dec, W, cfg)
    T = 617
    tiles = -(-T // 16)
    assert tiles % 2 == 1 and 4 * tiles > torch.cuda.get_device_properties(0).multi_processor_count >= 4 * -(-(T - 301) // 16)
    prompt = ref.rng_of(77).integers(0, 320, (4, T)).astype(np.int32)
    dec.reset(4)
    dec.prefill(prompt)
    one = dec.logits()
    _, logs = ref.Decoder(cfg, W).generate(prompt, 1)
    assert ref.err_inf(one, logs[0]) < 2e-2
    dec.reset(4)
    dec.prefill(prompt[:, :301])
    dec.prefill(prompt[:, 301:])
    assert ref.err_inf(dec.logits(), one) < 1e-3
    ctx.device_status()
    dec.free()


def test_rows_of_more_than_one_pass(ctx):
    """The bf16 planes of f32 rows beyond a gigabyte: two passes, of an odd total, added onto y."""
    import torch
    n, k, m = 272, 32768, 8203
    w = _weight(ctx, "q8", n, k)
    wd = w.dequant().double()
    x = torch.randn(m, k, device="cuda")
    y = torch.full((m, n + 8), 0.25, device="cuda")[:, :n]
    ctx.gemm_q4(w, x, out=y, flags=1)
    for r in (slice(0, 200), slice(4000, 4300), slice(m - 200, m)):
        want = x[r].double() @ wd.T + 0.25
        # K / 16 truncating tensor-core steps of 2^-24 of the running sum, as above: 1.3e-4 at the most
        assert float((y[r].double() - want).abs().max() / want.abs().max()) < 1.3e-4
    ctx.device_status()


def test_results_do_not_depend_on_the_call_before(ctx):
    """Back-to-back calls of several shapes share workspaces and overlap at their ends."""
    import torch
    ws = [_weight(ctx, f, n, k) for f, n, k in (("q4", 4096, 4096), ("q8", 1040, 992), ("q4", 272, 736))]
    calls = [(w, torch.randn(m, w.cols, device="cuda").to(d)) for w in ws for m, d in
             ((8, torch.bfloat16), (16, torch.float32), (101, torch.float32), (300, torch.bfloat16))]
    want = []
    for w, x in calls:
        want.append(ctx.gemm_q4(w, x).clone())
        torch.cuda.synchronize()
    for _ in range(3):
        got = [ctx.gemm_q4(w, x) for w, x in calls]
        for a, b in zip(got, want):
            assert torch.equal(a, b)
    ctx.device_status()


# Prompt attention tiles hold 128 (token, head) rows, here 64 tokens, and 64 keys: prompts one short of, at and one beyond a tile (and
# half of one), continued from an odd length, with a window that ends inside a tile; two sequences of unequal history are not
# possible (one length per call), so two equal ones.
@pytest.mark.parametrize("softcap,window", [(0.0, 0), (20.0, 0), (0.0, 21)])
@pytest.mark.parametrize("lens", [(31, 1), (32, 33), (65, 18), (17, 40), (63, 33), (64, 60)])
def test_prompt_in_two_calls_matches_the_teacher(ctx, lens, softcap, window):
    from cyb_b200 import qeng
    cfg = ref.DecoderConfig(layers=2, d=256, ffn=512, heads=4, kv_heads=2, vocab=320, attn_softcap=softcap, sliding_window=window)
    W = ref.make_decoder_weights(cfg, seed=5)
    dec = ctx.decoder(layers=2, d_model=256, ffn=512, heads=4, kv_heads=2, vocab=320, max_batch=2, max_seq=128,
                      attn_softcap=softcap, sliding_window=window)
    qeng.load_decoder_weights(dec, W, cfg)
    prompt = ref.rng_of(sum(lens)).integers(0, 320, (2, sum(lens))).astype(np.int32)
    dec.reset(2)
    dec.prefill(prompt[:, :lens[0]])
    dec.prefill(prompt[:, lens[0]:])
    want, logs = ref.Decoder(cfg, W).generate(prompt, 3)
    assert ref.err_inf(dec.logits(), logs[0]) < 2e-3
    assert np.array_equal(dec.decode(3), want)
    dec.free()


# Rows: one, a full launch and one over; V: less than one 8-row tile, a ragged last tile, and more than one round of CTAs;
# D: one chunk of 64, a cut one, many.  Bound: the activations are exact, a chunk of 64 products truncates at 4
# tensor-core steps (4 * 2^-24 of its partial sums) and the chunks are added with compensation: 2^-21 of the largest sum.
@pytest.mark.parametrize("v,d", [(5, 64), (1000, 200), (40001, 1032), (320, 4096)])
def test_lm_head_edges(ctx, v, d):
    import torch
    tb = (torch.randn(v, d, device="cuda") * 0.05).bfloat16()
    for m in (1, 5, 16, 17):
        x = torch.randn(m * d + 1, device="cuda")[1 if m == 5 else 0:][:m * d].view(m, d)
        y = ctx.lm_head(tb.view(torch.int16), x)
        want = x.double() @ tb.double().T
        assert float((y.double() - want).abs().max() / want.abs().max()) < 2.0 ** -21, (v, d, m)
    ctx.device_status()


# A tile of the prompt attention holds tokens that attend different keys.  Token 20's values overflow f16: the rows
# that do not attend it (before it, and with a window of 8 those from 28 on) give what they give without it.
@pytest.mark.parametrize("window", [0, 8])
def test_prompt_rows_do_not_see_infinite_values_they_do_not_attend(ctx, window):
    import torch
    from cyb_b200 import qeng
    cfg = ref.DecoderConfig(layers=1, d=256, ffn=512, heads=4, kv_heads=2, vocab=320, sliding_window=window)
    W = ref.make_decoder_weights(cfg, seed=5)
    q, s = W["layers"][0]["wv"]
    q, s = q.copy(), s.copy()
    q[:, :32], s[:, 0] = 8, 60000.0  # the first block only acts through column 0
    q[:, 0] = 15
    W["layers"][0]["wv"] = (q, s)
    dec = ctx.decoder(layers=1, d_model=256, ffn=512, heads=4, kv_heads=2, vocab=320, max_batch=1, max_seq=64, sliding_window=window)
    qeng.load_decoder_weights(dec, W, cfg)
    x = torch.randn(40, 256, device="cuda", generator=torch.Generator(device="cuda").manual_seed(3))
    x[:, 0] = 0.0
    plain = dec.layer(0, x, np.arange(40))
    assert bool(torch.isfinite(plain).all())
    x[20, 0] = 8.0
    got = dec.layer(0, x, np.arange(40))
    attends = range(20, 28 if window else 40)
    assert not bool(torch.isfinite(got[20]).any())
    rest = [r for r in range(40) if r not in attends]
    assert bool(torch.isfinite(got[rest]).all())
    # weights of one tile are summed in another order there: a few units of the two-term operands' 2^-17
    assert float((got[rest] - plain[rest]).abs().max() / plain.abs().max()) < 1e-4
    ctx.device_status()
    dec.free()


# The same for keys that overflow f16 (scores of both infinities, which sum to NaN): rows that attend them have no finite result, all
# others the same bits as without; and over several stages of keys with two tiles a CTA, an odd number of tiles, for values too.  Token
# 260 lies in the fifth stage of 64 keys; with a window of 116 the tiles of 16 tokens from 352 (every row attends the whole stage) and
# from 368 (some do not) share a CTA whose first stage is the one before, and go on to later ones.  Infinite values are summed key
# by key, in another order: a few units of the two-term operands' 2^-17.
@pytest.mark.parametrize("which,rows,at,window", [("wk", 40, 20, 0), ("wk", 40, 20, 8), ("wk", 617, 260, 0), ("wk", 617, 260, 116),
                                                  ("wv", 617, 260, 0), ("wv", 617, 260, 116)])
def test_prompt_rows_and_infinite_keys_or_values(ctx, which, rows, at, window):
    import torch
    from cyb_b200 import qeng
    heads, kv = (32, 4) if rows > 300 else (4, 2)
    tiles = -(-rows // (128 // (heads // kv)))
    if rows > 300:
        assert tiles % 2 == 1 and tiles * kv > torch.cuda.get_device_properties(0).multi_processor_count
    cfg = ref.DecoderConfig(layers=1, d=256, ffn=512, heads=heads, kv_heads=kv, vocab=320, sliding_window=window)
    W = ref.make_decoder_weights(cfg, seed=5, fmt="q8")
    q, s = W["layers"][0][which]
    q, s = q.copy(), s.copy()
    q[:, :32], s[:, 0] = 0, 60000.0  # the first block only acts through column 0
    q[:, 0] = 7
    W["layers"][0][which] = (q, s)
    dec = ctx.decoder(layers=1, d_model=256, ffn=512, heads=heads, kv_heads=kv, vocab=320, max_batch=1, max_seq=640, sliding_window=window)
    qeng.load_decoder_weights(dec, W, cfg)
    x = torch.randn(rows, 256, device="cuda", generator=torch.Generator(device="cuda").manual_seed(3))
    x[:, 0] = 0.0
    plain = dec.layer(0, x, np.arange(rows))
    assert bool(torch.isfinite(plain).all())
    x[at, 0] = 8.0
    got = dec.layer(0, x, np.arange(rows))
    end = min(rows, at + window) if window else rows
    assert not bool(torch.isfinite(got[at:end]).any())
    rest = [r for r in range(rows) if r < at or r >= end]
    if which == "wk":
        assert torch.equal(got[rest], plain[rest])
    else:
        assert float((got[rest] - plain[rest]).abs().max() / plain[rest].abs().max()) < 1e-4
    ctx.device_status()
    dec.free()


def test_lm_head_of_infinite_activations(ctx):
    """An infinite activation makes infinite logits (of the sign of the table's entry), NaN only where infinities meet."""
    import torch
    tb = (torch.randn(500, 136, device="cuda") * 0.05).bfloat16()
    x = torch.randn(4, 136, device="cuda")
    x[0, 3], x[1, 70], x[2, 5], x[2, 100] = float("inf"), -float("inf"), float("inf"), -float("inf")
    want = x @ tb.float().T
    y = ctx.lm_head(tb.view(torch.int16), x)
    special = ~torch.isfinite(want)
    assert bool(torch.isinf(want[:2]).all()) and bool(special[2].all()) and not bool(special[3].any())
    assert torch.equal(torch.nan_to_num(y[special], 7.0, 8.0, 9.0), torch.nan_to_num(want[special], 7.0, 8.0, 9.0))
    assert float((y[3] - want[3]).abs().max()) < 1e-5
    ctx.device_status()
