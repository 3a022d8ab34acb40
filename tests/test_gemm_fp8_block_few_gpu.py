"""The grouped block-fp8 GEMM for few rows per expert (``gemm_fp8_block_few_kernel``)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _blocks8(w):
    e, n, k = w.shape
    x = w.view(e, n // 128, 128, k // 128, 128)
    s = x.abs().amax((2, 4)) / 448.0
    return (x / s[:, :, None, :, None]).to(torch.float8_e4m3fn).view(e, n, k), s.contiguous()


def _wide(q, s):
    e, n, k = q.shape
    return (q.double().view(e, n // 128, 128, k // 128, 128) * s.double()[:, :, None, :, None]).view(e, n, k)


# rows per expert: none, one, a full tile, one more, several tiles; as few work items as one CTA's, and more than all CTAs have
@pytest.mark.parametrize("counts", [[1], [0, 16, 3, 0], [17, 64, 0, 65, 1, 130], [2] * 70])
@pytest.mark.parametrize("n,k", [(256, 128), (512, 768), (1536, 2048), (256, 4096)])
@pytest.mark.parametrize("block", [16, 32])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_against_64_bits(counts, n, k, block, dtype):
    from minisglang_rdna4_b200.ops import cuda as K
    from minisglang_rdna4_b200.ops import moe_kernels as MK

    g = torch.Generator("cuda")
    g.manual_seed(n + k + block)
    e = len(counts)
    owner = torch.repeat_interleave(torch.arange(e), torch.tensor(counts)).int()
    owner = owner[torch.randperm(len(owner))].cuda()
    t = len(owner)
    w, ws = _blocks8(torch.randn(e, n, k, generator=g, device="cuda") * 0.02)
    x = torch.randn(t, k, generator=g, device="cuda").to(dtype)
    _, pair_row, tile_expert, meta = MK.moe_align(owner.view(-1, 1), 0, e, block=block)
    rows = tile_expert.numel() * block
    xq, xs = MK.quantise_sorted("fp8_block", x, pair_row, rows, 1)
    at = pair_row.long()
    xd = (xq[at].double().view(t, k // 128, 128) * xs[at].double()[:, :, None]).view(t, k)
    want = torch.stack([xd[i] @ _wide(w[o:o + 1], ws[o:o + 1])[0].t() for i, o in enumerate(owner.tolist())])
    y = MK.gemm_fp8_block_few(xq, xs, w, ws, tile_expert, meta, block, dtype)[at]
    half = 2.0 ** -9 if dtype == torch.bfloat16 else 2.0 ** -12          # of a rounding to 16 bits
    assert float((y.double() - want).norm() / want.norm()) < half + 1e-5
    q, s = MK.gemm_fp8_block_few(xq, xs, w, ws, tile_expert, meta, block, dtype, glu=True)
    gate, up = y.double().chunk(2, -1)                                      # (as rounded)
    v = torch.nn.functional.silu(gate) * up
    got = (q[at].double().view(t, n // 256, 128) * s[at].double()[:, :, None]).view(t, n // 2)
    # half a step of e4m3, one rounding to 16 bits and the error of tanh.approx (2^-11 of SiLU's range)
    step = torch.maximum(v.abs(), 2.0 ** -6 * s[at].double().repeat_interleave(128, -1))
    assert float(((got - v).abs() / step).max()) <= 2.0 ** -4 + 2.0 ** -6
    assert float((got - v).norm() / v.norm()) < 2.0 ** -5 * 1.2
    assert K.gemm_fp8_block_status() == 0


# an even and an odd number of K blocks, one tile and several of a CTA
@pytest.mark.parametrize("m,n,k", [(5, 256, 512), (130, 1000, 640), (700, 8192, 256)])
def test_dense_scales_at_any_address(m, n, k):
    """Scales are single fp32 numbers: a view that begins in the middle of 8 or 16 bytes is read as any other."""
    from minisglang_rdna4_b200.ops import cuda as K

    g = torch.Generator("cuda")
    g.manual_seed(m)
    pad = -n % 128
    w, ws = _blocks8(torch.randn(1, n + pad, k, generator=g, device="cuda") * 0.02)
    w, ws = w[0, :n].contiguous(), ws[0]
    xq, xs = K.per_group_quant_fp8(torch.randn(m, k, generator=g, device="cuda").bfloat16(), 128)
    want = K.gemm_fp8_block(xq, xs, w, ws)
    full = (xq.double().view(m, -1, 128) * xs.double()[..., None]).view(m, k) @ _wide(
        torch.nn.functional.pad(w.view(torch.uint8), (0, 0, 0, pad)).view(torch.float8_e4m3fn)[None], ws[None])[0, :n].t()
    assert float((want.double() - full).norm() / full.norm()) < 2.0 ** -9 + 1e-5
    for off in (1, 2, 3):
        at = lambda t: torch.cat([t.new_zeros(off), t.reshape(-1)])[off:].view(t.shape)  # noqa: E731
        assert at(xs).data_ptr() % 16 == 4 * off
        assert torch.equal(K.gemm_fp8_block(xq, at(xs), w, at(ws)), want)


def test_a_layer_in_both_forms():
    from minisglang_rdna4_b200.ops import moe_kernels as MK

    g = torch.Generator("cuda")
    g.manual_seed(5)
    e, h, inter, k = 16, 1024, 512, 4
    w = _blocks8(torch.randn(e, 2 * inter, h, generator=g, device="cuda") * 0.03) + _blocks8(
        torch.randn(e, h, inter, generator=g, device="cuda") * 0.03)
    for t in (1, 5, 48, 49, 96):
        x = torch.randn(t, h, generator=g, device="cuda").bfloat16()
        wt, ids = torch.rand(t, e, generator=g, device="cuda").topk(k, -1)
        ids = ids.int()
        assert MK.few_rows_block(t * k, e, 2 * inter, h) > 0
        got = MK.moe_forward_quant("fp8_block", x, w, wt, ids)
        sp, pr, te, _ = MK.moe_align(ids, 0, e)
        want = MK._combine(MK.run_experts("fp8_block", MK._permute(x, sp, k), te, w, x.dtype), wt, pr, x, k)
        # the same sums and roundings in the same order: a verification step, which has more rows, agrees with decode steps
        assert torch.equal(got, want)


def test_what_it_does_not_take():
    from minisglang_rdna4_b200.ops import moe_kernels as MK

    assert MK.few_rows_block(8, 128, 1536, 2048) == 16
    for args in ((8, 128, 1536 + 128, 2048), (8, 128, 1536, 2048 + 64), (8, 128, 1536, 8192), (128 * 100, 128, 1536, 2048)):
        assert MK.few_rows_block(*args) == 0
