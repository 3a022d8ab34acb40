"""Row-wise kernels at the edges of their thread and vector counts: norms, gated activation and quantisers."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _rand(*shape, seed=0, dtype=torch.bfloat16):
    g = torch.Generator("cuda")
    g.manual_seed(seed + sum(shape))
    return torch.randn(*shape, generator=g, device="cuda").to(dtype)


def _same_rows8(got, want16):
    """e4m3 rows against the 16-bit rows they stand for: half a step of e4m3 (2^-4) at the row's scale."""
    q, s = got
    back = q.float() * s.reshape(s.shape[0], -1).repeat_interleave(q.shape[1] // max(1, s.numel() // s.shape[0]), 1)
    step = torch.maximum(want16.float().abs(), 2.0 ** -6 * s.reshape(s.shape[0], -1)[:, :1])
    assert float(((back - want16.float()).abs() / step).max()) <= 2.0 ** -4 * 1.02


# one vector a thread, two, and the last width of each block size; a width that ends inside a warp
@pytest.mark.parametrize("hidden", [8, 128, 1024, 1032, 2560, 4096, 4104, 8192, 8200, 16384])
@pytest.mark.parametrize("planes", [0, 1, 3, 4, 8])
def test_norm_widths(hidden, planes):
    from minisglang_rdna4_b200.ops import cuda as K

    if planes and hidden > 8192:
        pytest.skip("planes are summed up to 8192 columns")
    rows = 5
    res, w = _rand(rows, hidden, seed=1), _rand(hidden, seed=2)
    parts = _rand(max(planes, 1), rows, hidden, dtype=torch.float32)
    x = parts.sum(0).to(torch.bfloat16) if planes else _rand(rows, hidden)
    if planes:
        total = torch.zeros_like(parts[0])
        for p in parts:
            total = total + p
        x = total.to(torch.bfloat16)
    new = (x.float() + res.float()).to(torch.bfloat16)
    want = (new.double() * torch.rsqrt(new.double().square().mean(-1, keepdim=True) + 1e-6) * w.double())
    for quant in (False, True):
        r = res.clone()
        got = (K.rms_norm_planes(K.SplitPartial(parts, torch.bfloat16), r, w, 1e-6, quant=quant) if planes
               else K._rms(x, r, w, 1e-6, False, quant))
        assert torch.equal(r, new)
        if quant:
            _same_rows8(got, want.to(torch.bfloat16))
        else:   # one rounding to 16 bits of a product whose factors are good to fp32
            assert float(((got.double() - want).abs() / want.abs().clamp_min(1e-6)).max()) <= 2.0 ** -8 * 1.01


# the widest row whose norm sums planes, and wider ones
@pytest.mark.parametrize("hidden", [8192, 8200, 12288, 16384])
@pytest.mark.parametrize("rows", [1, 64, 128, 200])
@pytest.mark.parametrize("quant", [False, True])
def test_projection_and_norm_of_a_decode_step(hidden, rows, quant):
    """A row-parallel projection hands the norm behind it a sum that it can take, at every width a model may have."""
    from minisglang_rdna4_b200.core import Batch, Context, set_global_ctx
    from minisglang_rdna4_b200.layers.linear import RowParallelLinear
    from minisglang_rdna4_b200.layers.norm import RMSNorm
    from minisglang_rdna4_b200.parallel.comm import get_comm
    from minisglang_rdna4_b200.parallel.info import set_tp_info

    k = 512
    set_tp_info(0, 1)
    proj, norm = RowParallelLinear(k, hidden, torch.bfloat16, "cuda"), RMSNorm(hidden, 1e-6, torch.bfloat16, "cuda")
    proj.weight, norm.weight = _rand(hidden, k, seed=1), _rand(hidden, seed=2)
    x, res = _rand(rows, k, seed=3), _rand(rows, hidden, seed=4)
    get_comm().split_k_ok = True
    ctx = Context(page_size=16)
    set_global_ctx(ctx)
    with ctx.forward_batch(Batch(reqs=[], phase="decode")):
        got, new = norm.forward_fused(proj.forward(x), res.clone(), partial=True, quant=quant)
    y = x.double() @ proj.weight.double().t()
    # the projection and the sum with the residual are rounded to 16 bits each: half a step of eight significant bits, at most
    # 2^-8 of either; and fp32 sums of k products
    want = y + res.double()
    assert float(((new.double() - want).abs() - 2.0 ** -8 * (y.abs() + want.abs()) * 1.01).max()) <= 2.0 ** -12
    norm16 = (new.double() * torch.rsqrt(new.double().square().mean(-1, keepdim=True) + 1e-6) * norm.weight.double())
    if quant:
        _same_rows8((got.q, got.scale), norm16.to(torch.bfloat16))
    else:
        assert float(((got.double() - norm16).abs() / norm16.abs().clamp_min(1e-6)).max()) <= 2.0 ** -8 * 1.01


def test_a_norm_does_not_depend_on_the_rows_around():
    from minisglang_rdna4_b200.ops import cuda as K

    x, w = _rand(2100, 2560), _rand(2560, seed=3)
    whole = K.rms_norm(x, w, 1e-6)
    for a, b in ((0, 1), (7, 64), (1000, 1148)):
        assert torch.equal(K.rms_norm(x[a:b].contiguous(), w, 1e-6), whole[a:b])


@pytest.mark.parametrize("rows,hidden,runs", [(2047, 512, False), (2048, 512, True), (4095, 1024, False), (4096, 1016, True),
                                              (4096, 1032, False), (4100, 264, True)])
def test_many_short_rows_quantised_as_few(rows, hidden, runs):
    """A row's maximum does not depend on who takes it: the rows of a large call are those of small ones (``runs``: the form that the
    large one takes)."""
    from minisglang_rdna4_b200.ops import cuda as K

    x = _rand(rows, hidden)
    q, s = K.per_token_quant_fp8(x)
    for a in (0, 1000, rows - 9):
        part = K.per_token_quant_fp8(x[a:a + 9].contiguous())
        assert torch.equal(part[0].view(torch.uint8), q[a:a + 9].view(torch.uint8)) and torch.equal(part[1], s[a:a + 9])


@pytest.mark.parametrize("hidden", [2560, 2568, 4096, 4104, 8192, 8200])
@pytest.mark.parametrize("quant", [False, True])
def test_norm_without_a_residual(hidden, quant):
    from minisglang_rdna4_b200.ops import cuda as K

    x, w = _rand(7, hidden), _rand(hidden, seed=2)
    want = x.double() * torch.rsqrt(x.double().square().mean(-1, keepdim=True) + 1e-6) * w.double()
    got = K._rms(x, None, w, 1e-6, False, quant)
    if quant:
        _same_rows8(got, want.to(torch.bfloat16))
    else:   # one rounding to 16 bits of a product whose factors are good to fp32
        assert float(((got.double() - want).abs() / want.abs().clamp_min(1e-6)).max()) <= 2.0 ** -8 * 1.01


@pytest.mark.parametrize("rows,inter", [(1, 8), (2049, 1408), (2049, 2048), (2049, 2056), (3, 1024), (3, 1032), (2, 4096), (2049, 4104), (2049, 10240), (2049, 10248),
                                        (2, 12288), (2, 12296), (2, 20480), (2, 20488), (1, 28672)])
def test_gated_activation_quantised(rows, inter):
    from minisglang_rdna4_b200.ops import cuda as K

    x = _rand(rows, 2 * inter)
    _same_rows8(K.silu_and_mul_quant(x), K.act_and_mul(x))


def test_gated_activation_too_wide_is_refused():
    from minisglang_rdna4_b200.ops import cuda as K

    with pytest.raises(Exception):
        K.silu_and_mul_quant(_rand(1, 2 * 28680))


@pytest.mark.parametrize("hidden,group", [(8, 0), (248, 0), (256, 0), (264, 0), (512, 0), (520, 0), (8192, 0), (8200, 0), (16384, 0),
                                          (16392, 0), (2048, 128), (768, 128), (384, 96), (1024, 8), (1024, 512)])
def test_quantiser_groups(hidden, group):
    from minisglang_rdna4_b200.ops import cuda as K

    x = _rand(9, hidden)
    q, s = K.per_group_quant_fp8(x, group)
    amax = x.float().view(9, -1, group or hidden).abs().amax(-1)
    want = amax.clamp_min(1e-8) / torch.full_like(amax, 448)      # (a scalar divisor would be a product with its inverse)
    assert torch.equal(s.view(9, -1), want)
    _same_rows8((q.view(-1, group or hidden), s.reshape(-1)), x.view(-1, group or hidden))
