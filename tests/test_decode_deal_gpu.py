"""Decode attention with its tiles dealt evenly to the warps (``paged_decode_deal_kernel``), and rows that leave attention in
8 bits."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

PS = 16


def _case(lens, hq, hk, d, fp8, seed=0):
    from minisglang_rdna4_b200.ops import cuda as K

    g = torch.Generator("cuda")
    g.manual_seed(seed)
    pages = [-(-n // PS) for n in lens]
    total = sum(pages) + 1
    pool = K.make_pool_buffer(2, total + 1, hk, PS, d, torch.float8_e4m3fn if fp8 else torch.bfloat16, "cuda")
    pool[:, 1].copy_(torch.randn(pool[:, 1].shape, generator=g, device="cuda"))
    order = np.random.RandomState(seed).permutation(total)
    table = np.zeros((len(lens), max(pages + [1])), dtype=np.int32)
    at = 0
    for i, n in enumerate(pages):
        table[i, :n] = order[at:at + n]
        at += n
    q = torch.randn(len(lens), hq, d, generator=g, device="cuda").bfloat16()
    dev = lambda a: torch.tensor(a, dtype=torch.int32, device="cuda")  # noqa: E731
    return q, pool, dev(table), dev(list(range(len(lens) + 1))), dev(list(lens))


def _want(q, pool, table, lens, scale, ks, vs, window=0):
    hk = pool.shape[3]
    out = torch.zeros(q.shape, dtype=torch.float64, device="cuda")
    for i, n in enumerate(lens.tolist()):
        if n == 0:
            continue
        lo = max(0, n - window) if window else 0
        pages = table[i, :-(-n // PS)].long()
        k, v = (pool[w, 1][pages].double().transpose(1, 2).reshape(-1, hk, pool.shape[-1])[lo:n] * s.double()[None, :, None]
                for w, s in ((0, ks), (1, vs)))
        k, v = (t.permute(1, 0, 2).repeat_interleave(q.shape[1] // hk, 0) for t in (k, v))
        s = (q[i].double()[:, None] @ k.transpose(1, 2)) * scale
        out[i] = (s.softmax(-1) @ v)[:, 0]
    return out


def _run(c, fp8, window=0, scales=None, **kw):
    from minisglang_rdna4_b200.ops import cuda as K

    q, pool, table, cu, lens = c
    ks, vs = scales if fp8 else (None, None)
    return K.paged_attention(q, pool[0, 1], pool[1, 1], table, cu, lens, 0.1, k_scale=ks, v_scale=vs, max_q=1,
                             max_kv=table.shape[1] * PS, decode=True, window=window, **{"deal": True, **kw})


LENGTHS = {
    "one_tile": [1], "no_tiles": [0, 5, 0], "edge": [64, 65, 128, 129, 1], "alone": [700], "long": [40000],
    "ragged": [90, 3500, 64, 1, 1200, 65, 2500, 0, 333], "many": [(37 * i) % 500 + 1 for i in range(300)],
    "shortest": [64] * 40, "two": [20000, 70],
    # no request shared: more of them than warps, and fewer; the longest one just long enough to be shared, and a tile less
    "whole": [300 - i % 40 for i in range(96)], "whole_few": [200, 1, 64, 0, 150] * 8,
    "slack": [320, *[64] * 30], "slack_less": [288, *[64] * 30], "slack16": [224, *[64] * 30], "slack16_less": [192, *[64] * 30],
}


@pytest.mark.parametrize("name", sorted(LENGTHS))
@pytest.mark.parametrize("hq,hk,d,fp8", [(32, 8, 128, True), (8, 1, 128, False), (4, 4, 64, False), (24, 8, 128, True)])
def test_against_64_bits(name, hq, hk, d, fp8):
    from minisglang_rdna4_b200.ops import cuda as K

    c = _case(LENGTHS[name], hq, hk, d, fp8)
    scales = torch.linspace(0.5, 1.5, hk, device="cuda"), torch.linspace(1.25, 0.75, hk, device="cuda")
    one = torch.ones(hk, device="cuda")
    for window in (0, 100):
        got = _run(c, fp8, window=window, scales=scales)
        want = _want(c[0], c[1], c[2], c[4], 0.1, *(scales if fp8 else (one, one)), window)
        # weights are rounded to 16 bits (bf16: 2^-9) in front of the second product, and so is the result
        assert float((got.double() - want).norm()) <= 2.0 ** -8 * 1.5 * float(want.norm()) + 1e-12
        assert torch.equal(got, _run(c, fp8, window=window, scales=scales))
    assert K.attn_status() == 0


@pytest.mark.parametrize("name", ["ragged", "whole", "whole_few", "slack", "slack_less"])
def test_padding_rows_change_nothing(name):
    lens = LENGTHS[name]
    q, pool, table, cu, n = _case(lens, 32, 8, 128, True)
    one = torch.ones(8, device="cuda")
    alone = _run((q, pool, table, cu, n), True, scales=(one, one))
    pad = 7
    wide = (torch.cat([q, q[:pad]]), pool, torch.cat([table, table[:pad]]), torch.arange(len(lens) + pad + 1, device="cuda", dtype=torch.int32),
            torch.cat([n, torch.ones(pad, dtype=torch.int32, device="cuda")]))
    assert torch.equal(_run(wide, True, scales=(one, one))[:len(lens)], alone)


@pytest.mark.parametrize("kw", [dict(deal=True), dict(deal=False, splits=5)])
def test_rows_of_no_request_are_zero(kw):
    q, pool, table, cu, n = _case([100, 900], 32, 8, 128, True)
    one = torch.ones(8, device="cuda")
    wide = (torch.cat([q, q, q]), pool, table, cu, n)
    got = _run(wide, True, scales=(one, one), **kw)
    assert torch.equal(got[:2], _run((q, pool, table, cu, n), True, scales=(one, one), **kw)) and not bool(got[2:].any())
    q8, s = _run(wide, True, scales=(one, one), quant=True, **kw)
    assert not bool(q8.float()[2:].any()) and bool(torch.isfinite(s).all())


def test_gate_of_a_whole_and_of_a_shared_request():
    c = _case([30, 5000], 8, 2, 128, False)
    gate = torch.randn(2, 8 * 128, device="cuda").bfloat16()
    got = _run(c, False, gate=gate)
    want = _run(c, False).double() * torch.sigmoid(gate.double()).view(2, 8, 128)
    assert float((got.double() - want).norm() / want.norm()) < 2.0 ** -8


@pytest.mark.parametrize("hq,hk,fp8", [(32, 8, True), (64, 8, True), (4, 4, False), (40, 8, False)])
@pytest.mark.parametrize("kw", [dict(deal=True), dict(deal=False, splits=2), dict(deal=False, splits=16)])
def test_rows_in_8_bits_are_the_quantised_rows(hq, hk, fp8, kw):
    from minisglang_rdna4_b200.ops import cuda as K

    c = _case(LENGTHS["ragged"], hq, hk, 128, fp8)
    one = torch.ones(hk, device="cuda")
    rows = _run(c, fp8, scales=(one, one), **kw)
    want = K.per_token_quant_fp8(rows.view(rows.shape[0], -1))
    got = _run(c, fp8, scales=(one, one), quant=True, **kw)
    assert torch.equal(got[0].view(torch.uint8), want[0].view(torch.uint8)) and torch.equal(got[1], want[1])


@pytest.mark.parametrize("rows", [1, 2, 4, 5, 9, 18, 19, 37, 38, 148, 149])
@pytest.mark.parametrize("hq,hk", [(32, 8), (40, 8), (6, 6), (3, 1)])
@pytest.mark.parametrize("kw", [dict(deal=True), dict(deal=False, splits=3)])
def test_heads_of_a_row_over_several_ctas(rows, hq, hk, kw):
    """Few rows have their heads merged by several CTAs, many by one: the same sums."""
    lens = [600 + 37 * i % 300 for i in range(rows)]
    c = _case(lens, hq, hk, 128, False)
    got = _run(c, False, **kw)
    one = torch.ones(hk, device="cuda")
    want = _want(c[0], c[1], c[2], c[4], 0.1, one, one)
    assert float((got.double() - want).norm()) <= 2.0 ** -8 * 1.5 * float(want.norm())
    wide = _run(c, False, quant=True, **kw)       # (a CTA has the row)
    from minisglang_rdna4_b200.ops import cuda as K

    q, s = K.per_token_quant_fp8(got.view(rows, -1))
    assert torch.equal(wide[0].view(torch.uint8), q.view(torch.uint8)) and torch.equal(wide[1], s)


@pytest.mark.parametrize("kw", [dict(deal=True), dict(deal=False, splits=4)])
def test_a_workspace_at_any_address(kw):
    """The merge reads 16 bytes at a time: a workspace that begins elsewhere is not used."""
    c = _case(LENGTHS["ragged"], 32, 8, 128, False)
    want = _run(c, False, **kw)
    ws = torch.full((1 << 23,), float("nan"), device="cuda")
    assert torch.equal(_run(c, False, workspace=ws[1:], **kw), want) and bool(ws.isnan().all())
    assert torch.equal(_run(c, False, workspace=ws, **kw), want) and not bool(ws.isnan().all())


def test_graph_and_two_streams():
    c = _case(LENGTHS["ragged"], 32, 8, 128, True)
    one = torch.ones(8, device="cuda")
    run = lambda: _run(c, True, scales=(one, one))  # noqa: E731
    want = run()
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    outs = []
    for _ in range(10):
        outs.append(run())
        with torch.cuda.stream(side):
            outs.append(run())
    torch.cuda.synchronize()
    assert all(torch.equal(o, want) for o in outs)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.stream(side):
        run()
        side.synchronize()
        with torch.cuda.graph(graph, stream=side):
            y = run()
    for _ in range(3):
        y.zero_()
        torch.cuda.synchronize()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(y, want)


def test_a_pool_is_given_back():
    import gc

    before = torch.cuda.memory_allocated()
    c = _case([5000], 32, 8, 128, True)
    one = torch.ones(8, device="cuda")
    for deal in (True, False):
        _run(c, True, scales=(one, one), deal=deal)
    size = c[1].numel()
    del c
    gc.collect()
    torch.cuda.synchronize()
    assert torch.cuda.memory_allocated() - before < size


def test_what_it_does_not_cover():
    from minisglang_rdna4_b200.ops._lib import lib

    workers = lib().msgl_paged_decode_workers
    assert workers(4, 32, 8, 128, 16, 1, 0, 0) > 0
    for args in ((0, 32, 8, 128, 16, 1, 0, 0), (1025, 32, 8, 128, 16, 1, 0, 0), (4, 32, 2, 128, 16, 1, 0, 0),
                 (4, 30, 8, 128, 16, 1, 0, 0), (4, 32, 8, 128, 64, 1, 0, 0), (4, 32, 8, 64, 16, 1, 0, 0), (4, 32, 8, 256, 16, 0, 0, 0),
                 (4, 32, 8, 128, 16, 1, 1, 0), (4, 32, 8, 128, 16, 0, 1, 1), (4, 32, 8, 128, 16, 0, 0, 2)):
        assert workers(*args) == 0
