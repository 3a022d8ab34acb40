"""Expert rows: alignment in one launch and in several, rows quantised once per token, rows of no pair left out."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _rand(*shape, seed=0, dtype=torch.bfloat16):
    g = torch.Generator("cuda")
    g.manual_seed(seed + sum(shape))
    return torch.randn(*shape, generator=g, device="cuda").to(dtype)


# pairs at the edge of the one-launch alignment; experts of other ranks; an expert with most of the rows
@pytest.mark.parametrize("tokens,k,experts,start,local", [(1, 1, 1, 0, 1), (1, 8, 128, 0, 128), (48, 8, 128, 32, 64), (512, 8, 128, 0, 128),
                                                          (513, 8, 128, 0, 128), (700, 6, 512, 0, 512)])
def test_alignment(tokens, k, experts, start, local):
    from minisglang_rdna4_b200.ops import moe_kernels as MK

    g = torch.Generator("cuda")
    g.manual_seed(tokens)
    score = torch.rand(tokens, experts, generator=g, device="cuda")
    score[:, experts // 2] += 0.5
    ids = score.topk(k, -1).indices.int()
    sorted_pair, pair_row, tile_expert, meta = MK.moe_align(ids, start, local)
    here = (ids.long() - start).view(-1)
    ok = (here >= 0) & (here < local)
    count = torch.bincount(here[ok], minlength=local)
    tiles = (count + 127) // 128
    assert meta.tolist() == [int(tiles.sum()), int(tiles.sum()) * 128]
    want = torch.repeat_interleave(torch.arange(local, device="cuda"), tiles)
    assert torch.equal(tile_expert[:len(want)].long(), want) and bool((tile_expert[len(want):] == -1).all())
    assert bool((pair_row[~ok] == -1).all())
    rows = pair_row[ok].long()
    assert rows.unique().numel() == rows.numel() == int((sorted_pair >= 0).sum())
    assert torch.equal(sorted_pair[rows].long(), ok.nonzero().view(-1))
    assert torch.equal(tile_expert[rows // 128].long(), here[ok])


@pytest.mark.parametrize("kind", ["mxfp4", "fp8_block"])
@pytest.mark.parametrize("tokens,hidden,k", [(1, 128, 1), (5, 2048, 8), (130, 2176, 20), (33, 4096, 6)])
def test_quantised_expert_rows(kind, tokens, hidden, k):
    from minisglang_rdna4_b200.ops import cuda as K
    from minisglang_rdna4_b200.ops import moe_kernels as MK

    x = _rand(tokens, hidden)
    rows = tokens * k + 11
    pair_row = torch.randperm(rows, device="cuda")[:tokens * k].int()
    pair_row[::3] = -1
    q, s = MK.quantise_sorted(kind, x, pair_row, rows, k)
    want_q, want_s = MK.quantise_rows(kind, x)
    live = pair_row >= 0
    token = torch.arange(tokens * k, device="cuda") // k
    at = pair_row[live].long()
    assert torch.equal(q.view(torch.uint8)[at], want_q.view(torch.uint8)[token[live]]) and torch.equal(s[at], want_s[token[live]])


def test_rows_of_no_pair_are_left_out():
    from minisglang_rdna4_b200.ops import cuda as K

    x = _rand(70, 2 * 384)
    pair = torch.arange(70, device="cuda", dtype=torch.int32)
    pair[::2] = -1
    want, got = K.silu_and_mul_quant_group(x), K.silu_and_mul_quant_group(x, pair)
    assert torch.equal(got[0].view(torch.uint8)[1::2], want[0].view(torch.uint8)[1::2]) and torch.equal(got[1][1::2], want[1][1::2])
