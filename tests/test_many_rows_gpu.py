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


# One-term operands: the smallest and largest token tiles with two accumulators and with one, remainders of both, tiles cut
# along K and whole ones, more tiles than CTA pairs.  Against operands rounded to bf16, only the sums differ: bound as above.
@pytest.mark.parametrize("m,n,k", [(256, 272, 736), (257, 4096, 992), (320, 1040, 4096), (416, 4112, 2048), (777, 2064, 4064), (2049, 4096, 544)])
def test_prompt_rows_and_widths(ctx, m, n, k):
    import torch
    w = _weight(ctx, "q4", n, k)
    wd = w.dequant().bfloat16().double()
    for dt in DT[:2]:
        x = torch.randn(m, k, device="cuda").to(getattr(torch, dt))
        y = torch.full((m, n + 8), 0.25, device="cuda")[:, :n]
        acc = m % 2
        ctx.gemm_q4(w, x, out=y, flags=acc)
        want = x.bfloat16().double() @ wd.T + (0.25 if acc else 0.0)
        err = float((y.double() - want).abs().max() / want.abs().max())
        assert err < 3e-5, (m, n, k, dt, err)
    ctx.device_status()


# Query heads per kv head: one, the most there are, and counts that do not divide the 64 rows of a prompt attention tile
# (its last rows stay empty); tiles then hold 64, 8, 21, 12, 10 and 9 tokens.
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


# Prompt attention tiles hold 64 (token, head) rows and 32 keys: prompts one short of, at and one beyond a tile, continued
# from an odd length, with a window that ends inside a tile, two sequences of unequal history are not possible (one length
# per call), so two equal ones.
@pytest.mark.parametrize("softcap,window", [(0.0, 0), (20.0, 0), (0.0, 21)])
@pytest.mark.parametrize("lens", [(31, 1), (32, 33), (65, 18), (17, 40)])
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


# A 64-row tile of the prompt attention holds tokens that attend different keys.  Token 20's values overflow f16: the rows
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
