"""Calls on several streams of one context and inside stream captures: whose working memory a call uses, how long it stays."""
import numpy as np
import pytest

from oracle import ref

pytestmark = pytest.mark.gpu


@pytest.fixture
def fresh(ctx):
    """A context that holds no working memory yet (the session's one has loaded the kernels)."""
    from cyb_b200 import qeng
    c = qeng.Context(0)
    yield c
    c.device_status()
    c.close()


def _weight(ctx, fmt, n, k):
    import torch
    g = torch.Generator(device="cuda")
    g.manual_seed(n + k)
    if fmt == "q4k":
        return ctx.pack_q4k(ref.make_q4k(ref.rng_of(7), n, k)[2], n, k)
    w = torch.randn(n, k, device="cuda", generator=g) * 0.05
    return ctx.quantize_q4(w) if fmt == "q4" else ctx.quantize_q8(w)


# one shape of every kernel and of every buffer it needs: slices without planes, planes, block sums, tiles cut along K
SHAPES = [("q4", 3, "bfloat16"), ("q4", 4, "bfloat16"), ("q8", 8, "float32"), ("q4k", 16, "float16"), ("q4", 101, "float32"),
          ("q4", 300, "bfloat16"), ("q4", 300, "float32")]
N, K = 2064, 1280


# three and four rows over tall matrices (40000 values of activations and more) need slices, too
@pytest.mark.parametrize("fmt,m,dt,n,k", [s + (N, K) for s in SHAPES] + [("q4", 4, "float32", 1040, 10016), ("q8", 3, "float16", 272, 13344)])
def test_captured_matmul_has_a_workspace_of_its_own(ctx, fresh, fmt, m, dt, n, k):
    """The first call of the context is captured; its graph is replayed beside calls on the stream that did not capture,
    and after calls that outgrow and displace every stream's buffers."""
    import torch
    w0 = _weight(ctx, fmt, n, k)
    w = _weight(fresh, fmt, n, k)
    x = torch.randn(m, k, device="cuda").to(getattr(torch, dt))
    x2 = torch.randn(m, k, device="cuda").to(getattr(torch, dt))
    want, want2 = ctx.gemm_q4(w0, x), ctx.gemm_q4(w0, x2)  # loads the kernels, too
    y = torch.zeros(m, n, device="cuda")
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        fresh.gemm_q4(w, x, out=y)
    for _ in range(20):
        g.replay()
        y2 = fresh.gemm_q4(w, x2)
    torch.cuda.synchronize()
    assert torch.equal(y, want) and torch.equal(y2, want2)
    side = torch.cuda.Stream()
    for _ in range(20):  # side by side
        with torch.cuda.stream(side):
            g.replay()
        y2 = fresh.gemm_q4(w, x2)
    torch.cuda.synchronize()
    assert torch.equal(y, want) and torch.equal(y2, want2)
    big = torch.randn(4 * m, k, device="cuda").to(getattr(torch, dt))
    for s in [torch.cuda.Stream() for _ in range(10)]:
        with torch.cuda.stream(s):
            fresh.gemm_q4(w, big)
    fresh.gemm_q4(w, big)
    torch.cuda.synchronize()
    y.zero_()
    g.replay()
    torch.cuda.synchronize()
    assert torch.equal(y, want)


def test_row_count_that_only_the_streaming_matmul_takes(ctx, fresh):
    """8 rows over a K too wide for the batch kernel's slices: quantised activation images, on two streams and in a graph."""
    import torch
    n, k = 64, 10 ** 6 + 32
    w = _weight(fresh, "q4", n, k)
    xs = [torch.randn(8, k, device="cuda") for _ in range(3)]
    want = [ctx.gemm_q4(w, x) for x in xs]
    exact = w.dequant().double()
    for x, y in zip(xs, want):  # activations in 15 bits per block
        assert float((y.double() - x.double() @ exact.T).norm() / y.double().norm()) < 3e-4
    y = torch.zeros_like(want[0])
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        fresh.gemm_q4(w, xs[0], out=y)
    streams = [torch.cuda.Stream() for _ in range(3)]
    outs = [[], []]
    for _ in range(20):
        with torch.cuda.stream(streams[0]):
            g.replay()
        for i in (0, 1):
            with torch.cuda.stream(streams[1 + i]):
                outs[i].append(fresh.gemm_q4(w, xs[1 + i]))
    torch.cuda.synchronize()
    assert torch.equal(y, want[0])
    for i in (0, 1):
        assert all(torch.equal(o, want[1 + i]) for o in outs[i])


def test_weight_shared_by_contexts_of_two_threads(ctx, fresh):
    """Two threads, each with its context and stream, over one weight: every call works out or looks up what the weight keeps
    per row count (more row counts than it keeps)."""
    import threading
    import torch
    w = _weight(ctx, "q4", N, K)
    rows = (5, 6, 8, 9, 12, 16, 24, 32)
    xs = [torch.randn(m, K, device="cuda").to(torch.bfloat16) for m in rows]
    want = [ctx.gemm_q4(w, x) for x in xs]
    torch.cuda.synchronize()
    bad = []

    def work(c, order):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                for i in order * 40:
                    y = c.gemm_q4(w, xs[i])
                    torch.cuda.current_stream().synchronize()
                    if not torch.equal(y, want[i]):
                        bad.append(rows[i])
        except Exception as e:  # noqa: BLE001  reported by the assertion
            bad.append(e)

    n = len(rows)
    threads = [threading.Thread(target=work, args=a) for a in ((ctx, list(range(n))), (fresh, [(3 * i) % n for i in range(n)]))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad, bad


def test_two_streams_of_one_capture(ctx):
    """Branches of one graph run side by side: they may not share a workspace either, nor may a second call outgrow what the
    first one of the capture uses."""
    import torch
    w = _weight(ctx, "q4", N, K)
    xs = [torch.randn(m, K, device="cuda") for m in (40, 40, 101)]
    want = [ctx.gemm_q4(w, x) for x in xs]
    ys = [torch.zeros_like(t) for t in want]
    torch.cuda.synchronize()
    side = torch.cuda.Stream()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        side.wait_stream(torch.cuda.current_stream())
        ctx.gemm_q4(w, xs[0], out=ys[0])
        ctx.gemm_q4(w, xs[2], out=ys[2])
        with torch.cuda.stream(side):
            ctx.gemm_q4(w, xs[1], out=ys[1])
        torch.cuda.current_stream().wait_stream(side)
    for _ in range(10):
        for t in ys:
            t.zero_()
        g.replay()
        torch.cuda.synchronize()
        assert all(torch.equal(a, b) for a, b in zip(ys, want))
    ctx.device_status()


def test_working_memory_of_dropped_graphs_is_used_again(fresh):
    import torch
    w = _weight(fresh, "q4", 4096, 4096)
    x, y = torch.randn(2048, 4096, device="cuda"), torch.zeros(2048, 4096, device="cuda")
    fresh.gemm_q4(w, x, out=y)

    def once():
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            fresh.gemm_q4(w, x, out=y)  # 16 MB of bf16 rows
        g.replay()
        torch.cuda.synchronize()
        del g

    once()
    before = torch.cuda.mem_get_info()[0]
    for _ in range(16):
        once()
    assert before - torch.cuda.mem_get_info()[0] < 64 << 20


def test_decoder_moved_to_another_stream(ctx):
    """The captured decode step keeps working memory of its own when the decoder changes streams: matmuls still running on
    the stream it left do not disturb it."""
    import torch
    from cyb_b200 import qeng
    cfg = ref.DecoderConfig(layers=2, d=256, ffn=512, heads=4, kv_heads=2, vocab=320)
    W = ref.make_decoder_weights(cfg, seed=5)
    dec = ctx.decoder(layers=2, d_model=256, ffn=512, heads=4, kv_heads=2, vocab=320, max_batch=8, max_seq=96)
    qeng.load_decoder_weights(dec, W, cfg)
    prompt = ref.rng_of(8).integers(0, 320, (8, 5)).astype(np.int32)
    want, _ = ref.Decoder(cfg, W).generate(prompt, 24)
    w = _weight(ctx, "q4", 4096, 4096)
    x = torch.randn(16, 4096, device="cuda")
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    with torch.cuda.stream(b):
        ctx.gemm_q4(w, x)
    with torch.cuda.stream(a):
        dec.use_current_stream()
    dec.reset(8)
    dec.prefill(prompt)
    got = [dec.decode(4)]
    with torch.cuda.stream(b):
        dec.use_current_stream()
    for _ in range(5):
        with torch.cuda.stream(a):
            for _ in range(200):
                ctx.gemm_q4(w, x)
        got.append(dec.decode(4))
    torch.cuda.synchronize()
    assert np.array_equal(np.concatenate(got, 1), want)
    ctx.device_status()
    dec.free()


# More (sequence, kv head) pairs than the cluster form takes (74 on 148 SMs): the fixed splits and their scratch.
def _attn_case(ctx, seed, B=20, hi=600):
    import torch
    lens, q, ks, vs, pool_np, table = ref.config4(seed=seed, B=B, lo=hi // 2, hi=hi)
    pool = ctx.kv_pool(pool_np.shape[0], pool_np.shape[1])
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    pool.tensor().copy_(t(pool_np))
    return (pool, t(q), t(table), t(lens)), ref.attn_decode(q, ks, vs)


def test_attention_of_many_sequences_on_two_streams(ctx, fresh):
    """Calls that overlap keep their arrival counters and partials apart, also where one grows its own, and in a graph."""
    import torch
    cases = [_attn_case(fresh, 1), _attn_case(fresh, 2), _attn_case(fresh, 3, B=24)]
    for args, _ in cases:  # loads the kernels
        ctx.attn_decode(*args)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    held = torch.zeros_like(cases[0][0][1], dtype=torch.float32)
    with torch.cuda.graph(g):
        fresh.attn_decode(*cases[0][0], out=held)
    streams = [torch.cuda.Stream() for _ in range(3)]
    outs = [[], [], []]
    for _ in range(30):
        for i, s in enumerate(streams[:2]):
            with torch.cuda.stream(s):
                outs[i].append(fresh.attn_decode(*cases[i][0]))
        with torch.cuda.stream(streams[2]):
            g.replay()
    with torch.cuda.stream(streams[0]):
        outs[2].append(fresh.attn_decode(*cases[2][0]))
    torch.cuda.synchronize()
    assert ref.err_inf(held.cpu().numpy(), cases[0][1]) < 1e-4
    for (_, want), got in zip(cases, outs):
        assert ref.err_inf(got[0].cpu().numpy(), want) < 1e-4
        # the order in which the splits are merged is fixed: every call gives the same bits
        assert all(torch.equal(o, got[0]) for o in got)
    for args, _ in cases:
        args[0].free()


def test_calls_that_find_no_memory_for_their_workspace(ctx, fresh):
    """8-bit, K-quant and short 4-bit matmuls and the attention of many sequences need none in passes or clusters: a full
    device makes them slower, not fail, and the failed allocation is not reported by the next launch."""
    import torch
    n = 1040
    cases = []
    for fmt, m, k in (("q8", 4096, 8192), ("q4k", 2048, 8192), ("q4", 255, 65536)):  # planes of 64 MB and more
        w = _weight(fresh, fmt, n, k)
        x = torch.randn(m, k, device="cuda")
        cases.append((w, x, ctx.gemm_q4(w, x), torch.empty(m, n, device="cuda")))
        for r in (1, 4, 15, 16):  # loads the kernels of the passes
            ctx.gemm_q4(w, x[:r])
    args, want = _attn_case(fresh, 4)
    held = ctx.attn_decode(*args)
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    hog = []
    for part in (1 << 30, 1 << 26, 1 << 24):  # down to 32..48 MB, which kernels still to be loaded may need
        while torch.cuda.mem_get_info()[0] > part + (32 << 20):
            hog.append(torch.empty(part, dtype=torch.uint8, device="cuda"))
    assert torch.cuda.mem_get_info()[0] < 56 << 20
    for w, x, y, out in cases:
        fresh.gemm_q4(w, x, out=out)
    fresh.attn_decode(*args, out=held)
    torch.cuda.synchronize()
    hog.clear()
    torch.cuda.empty_cache()
    for w, x, y, out in cases:
        # activations in 15 bits per block against bf16 pairs
        assert float((out - y).norm() / y.norm()) < 3e-4, w.fmt
    assert ref.err_inf(held.cpu().numpy(), want) < 1e-4
    args[0].free()


def _fill_device():
    """Blocks of device memory that leave none of 512 bytes (past torch's cache, which keeps to whole megabytes)."""
    import ctypes
    rt = ctypes.CDLL("libcudart.so.12")
    held, size = [], 1 << 36
    while size >= 512:
        p = ctypes.c_void_p()
        if rt.cudaMalloc(ctypes.byref(p), ctypes.c_size_t(size)) == 0:
            held.append(p)
        else:
            rt.cudaGetLastError()
            size >>= 1
    return lambda: [rt.cudaFree(p) for p in held]


def test_few_rows_of_tall_matrices_that_find_no_memory(ctx, fresh):
    """Three and four rows over a tall matrix, and the layers of four sequences with such a down projection, go through the integer
    kernel (15 bits per block) where there is no room for the slices of the other one (17 bits), and through that one again
    afterwards."""
    import torch
    from cyb_b200 import qeng
    calls = []
    for fmt, m, n, k in (("q4", 4, 1040, 10016), ("q8", 3, 1040, 13344)):
        w, small = _weight(fresh, fmt, n, k), _weight(ctx, fmt, n, 9984)
        x = torch.randn(m, k, device="cuda")
        calls.append((w, x, ctx.gemm_q4(w, x), torch.empty(m, n, device="cuda")))
        ctx.gemm_q4(small, x[:, :9984])  # loads the integer kernel
    cfgs = [ref.DecoderConfig(layers=1, d=256, ffn=f, heads=4, kv_heads=2, vocab=320) for f in (9984, 10240)]
    prompt = ref.rng_of(4).integers(0, 320, (4, 1)).astype(np.int32)
    decs = []
    for c, cfg in zip((ctx, fresh), cfgs):
        decs.append(c.decoder(layers=1, d_model=256, ffn=cfg.ffn, heads=4, kv_heads=2, vocab=320, max_batch=4, max_seq=32))
        W = ref.make_decoder_weights(cfg, seed=8)
        qeng.load_decoder_weights(decs[-1], W, cfg)
        decs[-1].reset(4)
    decs[0].prefill(prompt)
    decs[0].logits()
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    release = _fill_device()
    try:
        for w, x, y, out in calls:
            fresh.gemm_q4(w, x, out=out)
        decs[1].prefill(prompt)
        torch.cuda.synchronize()
        without = decs[1].logits()
    finally:
        release()
    for w, x, y, out in calls:
        assert 0.0 < float((out - y).norm() / y.norm()) < 3e-4, w.fmt
        assert torch.equal(fresh.gemm_q4(w, x), y)
    decs[1].reset(4)
    decs[1].prefill(prompt)
    _, logs = ref.Decoder(cfgs[1], W).generate(prompt, 1)
    assert ref.err_inf(without, logs[0]) < 2e-3 and ref.err_inf(decs[1].logits(), logs[0]) < 2e-3
    assert not np.array_equal(decs[1].logits(), without)
    for d in decs:
        d.free()
