"""The GEMM of decode steps (``csrc/gemm_stream.cu``): weights dealt to the CTAs in equal ranges of K blocks."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu

KINDS = {"f16": 0, "bf16": 1, "f8": 2, "mxf4": 3}


def _operands(kind, m, n, k):
    from minisglang_rdna4_b200.ops import cuda as K
    from minisglang_rdna4_b200.ops import ref as R
    from minisglang_rdna4_b200.quant import mxfp4

    g = torch.Generator("cuda")
    g.manual_seed(m * 7 + n + k)
    x = torch.randn(m, k, generator=g, device="cuda")
    w = torch.randn(n, k, generator=g, device="cuda") * 0.02
    if kind in ("f16", "bf16"):
        dt = torch.float16 if kind == "f16" else torch.bfloat16
        return (x.to(dt), w.to(dt), None, None, None), x.to(dt).double() @ w.to(dt).double().t()
    xq, xs = K.per_token_quant_fp8(x.bfloat16())
    xd = xq.double() * xs.double()[:, None]
    if kind == "f8":
        s = (w.abs().amax(-1) / 448).contiguous()
        wq = (w / s[:, None]).to(torch.float8_e4m3fn)
        return (xq, wq, xs, s, None), xd @ (wq.double() * s.double()[:, None]).t()
    packed, sf = mxfp4.quantize_mxfp4(w)
    pad = (-k % 128) // 2
    return (xq, torch.nn.functional.pad(packed, (0, pad)), xs, None, mxfp4.pack_sf_atoms(sf)), xd @ R.dequant_mxfp4(packed, sf).double().t()


# one tile and one K block; tiles with rows past N; K that ends inside a block; as many tiles as CTAs and a few more;
# a tile shared by the most CTAs; rows at the edges of the column counts
@pytest.mark.parametrize("m,n,k", [(1, 128, 128), (16, 136, 512), (17, 1000, 1216), (32, 2560, 9728), (33, 6144, 2560),
                                   (64, 19456, 1024), (65, 128, 4096), (128, 2560, 4096)])
@pytest.mark.parametrize("kind", sorted(KINDS))
def test_against_64_bits(kind, m, n, k):
    from minisglang_rdna4_b200.ops import cuda as K

    (x, w, xs, ws, sf), want = _operands(kind, m, n, k)
    bias = torch.randn(n, device="cuda").bfloat16()
    run = lambda planes, dt, b: K._gemm_stream(KINDS[kind], x, w, m, n, k, dt, xs, ws, b, sf, planes)  # noqa: E731
    # fp32 sums of K products: the error of one is at most K/2 ulp of the sum of their magnitudes, on average its root
    tol = 2.0 ** -23 * k ** 0.5 + 2.0 ** -22
    y = run(False, torch.float32, None)
    assert float((y.double() - want).norm() / want.norm()) < tol
    assert torch.equal(y, run(False, torch.float32, None))
    parts = run(True, torch.float32, bias)
    assert 1 <= parts.planes.shape[0] <= K.STREAM_PLANES and parts.planes.shape[1:] == (m, n)
    full = want + bias.double()
    assert float((parts.planes.double().sum(0) - full).norm() / full.norm()) < tol
    y16 = run(False, torch.bfloat16, bias)
    assert float((y16.double() - full).norm() / full.norm()) < 2.0 ** -8
    assert K.gemm_status() == 0


def test_a_row_is_the_same_in_every_batch():
    from minisglang_rdna4_b200.ops import cuda as K

    n, k = 2560, 2048
    (x, w, *_), _ = _operands("bf16", 128, n, k)
    run = lambda m, planes: K._gemm_stream(1, x[:m].contiguous(), w, m, n, k, torch.float32, None, None, None, None, planes)  # noqa: E731
    whole, parts = run(128, False), run(128, True).planes
    for m in (1, 16, 31, 64, 100):
        assert torch.equal(run(m, False), whole[:m]) and torch.equal(run(m, True).planes, parts[:, :m])


def test_calls_on_two_streams_have_counters_of_their_own():
    from minisglang_rdna4_b200.ops import cuda as K

    (x, w, *_), want = _operands("bf16", 8, 2560, 4096)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    outs = []
    for _ in range(20):
        outs.append(K._gemm_stream(1, x, w, 8, 2560, 4096, torch.float32, None, None, None, None, False))
        with torch.cuda.stream(side):
            outs.append(K._gemm_stream(1, x, w, 8, 2560, 4096, torch.float32, None, None, None, None, False))
    torch.cuda.synchronize()
    assert all(torch.equal(o, outs[0]) for o in outs)


def _shared_tiles(n, k):
    """A product whose tiles several CTAs share, and its result."""
    from minisglang_rdna4_b200.ops import cuda as K

    (x, w, *_), _ = _operands("bf16", 8, n, k)
    run = lambda: K._gemm_stream(1, x, w, 8, n, k, torch.float32, None, None, None, None, False)  # noqa: E731
    return run, run()


def _captured(run, stream, pool=None):
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, pool=pool, stream=stream):
        y = run()
    return graph, y


@pytest.mark.parametrize("warm", [True, False])
def test_graphs_of_one_pool_in_any_order(warm):
    """A graph finds its counters at zero whatever ran before it: the pool's memory belongs to the other graphs too, and the
    graph that was captured first need not be the one that is replayed first."""
    run, want = _shared_tiles(2560, 4096)
    stream = torch.cuda.Stream()
    torch.cuda.synchronize()
    if warm:
        with torch.cuda.stream(stream):
            run()
        stream.synchronize()
    with torch.cuda.stream(stream):
        # its scratch is free again, and may be anybody's, when the others are captured
        spoil, _ = _captured(lambda: torch.full((1 << 17,), 7, dtype=torch.int32, device="cuda").sum(), stream)
        graphs = [_captured(run, stream, spoil.pool()) for _ in range(2)]
    torch.cuda.synchronize()
    for at in (None, 1, None, 0, None, 1, 1, 0, None, None, 0):
        if at is None:
            spoil.replay()
            continue
        graph, y = graphs[at]
        y.fill_(float("nan"))
        torch.cuda.synchronize()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(y, want)


def test_graphs_of_one_stream_side_by_side():
    run, want = _shared_tiles(256, 2048)      # (few CTAs: two graphs fit on the GPU at once)
    stream = torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(stream):
        run()
        stream.synchronize()
        pairs = [_captured(lambda: [run() for _ in range(50)], stream) for _ in range(2)]
    torch.cuda.synchronize()
    for _ in range(20):
        for _, ys in pairs:
            for y in ys:
                y.fill_(float("nan"))
        sides = [torch.cuda.Stream() for _ in pairs]
        for (graph, _), s in zip(pairs, sides):
            s.wait_stream(torch.cuda.current_stream())
            with torch.cuda.stream(s):
                graph.replay()
        torch.cuda.synchronize()
        assert all(torch.equal(y, want) for _, ys in pairs for y in ys)


def test_counters_of_many_streams_and_captures(monkeypatch):
    from minisglang_rdna4_b200.ops import cuda as K

    monkeypatch.setattr(K, "_STREAM_COUNTERS", {})
    monkeypatch.setattr(K, "_CAPTURE_COUNTERS", {})
    at = [0, 0]
    monkeypatch.setattr(K, "_stream", lambda: at[0])
    monkeypatch.setattr(K, "_capture_id", lambda stream: at[1])
    first = K._stream_counters("cuda", 8)
    for at[0] in range(1, 3 * K.STREAM_COUNTER_SETS):
        assert K._stream_counters("cuda", 8) is K._stream_counters("cuda", 9)
        at[0], keep = 0, at[0]
        assert K._stream_counters("cuda", 8) is first     # a stream in use keeps its set
        at[0] = keep
    assert len(K._STREAM_COUNTERS) == K.STREAM_COUNTER_SETS
    at[:] = [5, 1]
    small = K._stream_counters("cuda", 8)
    large = K._stream_counters("cuda", 10 ** 5)
    assert large.numel() >= 10 ** 5 and not bool(large.any())
    assert K._CAPTURE_COUNTERS[("cuda", 5)][1][0] is small        # both stay while their capture goes on
    at[1] = 2
    assert K._stream_counters("cuda", 8) is not small and len(K._CAPTURE_COUNTERS[("cuda", 5)][1]) == 1


def test_which_products_it_takes(monkeypatch):
    from minisglang_rdna4_b200.ops import cuda as K

    for kind in range(4):
        for n in (8, 128, 1000, 2560, 12288, 18944, 18952, 151936):
            for k in (128, 1216, 2048, 4096, 28672):
                rows = K._stream_rows(kind, n, k, False)
                assert 0 <= rows <= (64 if n * k * (2, 2, 1, 0.5)[kind] >= 48 << 20 else 32)
                assert rows == 0 or k >= 2048 or n > 148 * 128
                assert K._stream_rows(kind, n, k, True) == (128 if k >= 2048 else 0)
    # few tiles and a long chain; as many tiles as SMs; a short chain
    assert K._stream_rows(1, 2560, 9728, False) == 32 and K._stream_rows(1, 4096, 12288, False) == 64
    assert K._stream_rows(3, 16384, 4096, False) < 16 and K._stream_rows(2, 1000, 1216, False) == 0
    taken = []
    monkeypatch.setattr(K, "_gemm_stream", lambda kind, a, b, m, *r: taken.append(m) or torch.empty(m, b.shape[0], device="cuda"))
    w = torch.zeros(2560, 9728, device="cuda", dtype=torch.bfloat16)
    for m in (0, 1, 32, 33):
        K.gemm(torch.zeros(m, 9728, device="cuda", dtype=torch.bfloat16), w, None, torch.float32, few=True)
    assert taken == [1, 32]


def test_operands_it_does_not_take_are_refused():
    from minisglang_rdna4_b200.ops import cuda as K
    from minisglang_rdna4_b200.ops._lib import lib

    x, w = torch.randn(4, 128, device="cuda").bfloat16(), torch.randn(256, 128, device="cuda").bfloat16()
    out = torch.empty(4, 256, device="cuda")
    args = lambda m, n, lda: lib().msgl_gemm_stream(1, x.data_ptr(), lda, w.data_ptr(), out.data_ptr(), n, m, n, 128, None, None,  # noqa: E731
                                                    None, 0, None, 2, 1, 1, None, None, K._stream())
    assert args(129, 256, 128) != 0 and args(4, 250, 128) != 0 and args(4, 256, 129) != 0 and args(0, 256, 128) != 0
    most = ctypes.c_int()
    for kind, n, k in ((3, 2560, 9728), (1, 8192, 28672), (2, 128, 128)):
        ctas = lib().msgl_gemm_stream_plan(kind, n, k, 8, ctypes.addressof(most))
        assert 1 <= ctas <= torch.cuda.get_device_properties(0).multi_processor_count and 1 <= most.value <= 8
