"""Arg-max by a cluster of CTAs per row."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _rand(*shape, seed=0, dtype=torch.bfloat16):
    g = torch.Generator("cuda")
    g.manual_seed(seed + sum(shape))
    return torch.randn(*shape, generator=g, device="cuda").to(dtype)


@pytest.mark.parametrize("vocab", [1, 5, 2047, 16383, 16384, 16397, 151936])
@pytest.mark.parametrize("rows", [1, 37, 75, 300])
def test_argmax_of_shares(vocab, rows):
    from minisglang_rdna4_b200.ops import cuda as K

    x = _rand(rows, vocab, dtype=torch.float32)
    top = torch.randint(0, vocab, (rows,), device="cuda")
    x[torch.arange(rows, device="cuda"), top] = 50.0
    x[0, :] = 7.0                                        # ties: the first one counts
    x[-1, vocab - 1] = 100.0                             # the last share's last value
    assert torch.equal(K.argmax(x).long(), x.argmax(-1))
    x[0] = float("-inf")
    assert int(K.argmax(x)[0]) == 0
    wide = torch.full((rows, vocab + 3), 1000.0, device="cuda")
    wide[:, :vocab] = x
    assert torch.equal(K.argmax(wide[:, :vocab]).long(), torch.where(torch.isinf(x.amax(-1)), 0, x.argmax(-1)))


# on both sides of every line of the plan
@pytest.mark.parametrize("vocab,rows", [(v, r) for v in (16383, 16384, 65535, 65536) for r in
                                        (18, 19, 37, 38, 50, 51, 74, 75, 148, 149, 222, 223, 296, 297)])
def test_argmax_of_any_number_of_rows(vocab, rows):
    from minisglang_rdna4_b200.ops import cuda as K

    x = _rand(rows, vocab, dtype=torch.float32)
    at = torch.arange(rows, device="cuda")
    x[at, (at * 7919) % vocab] = 60.0
    assert torch.equal(K.argmax(x).long(), (at * 7919) % vocab)


def test_beside_other_work():
    """CTAs of a cluster that start far apart, behind and beside kernels that hold most of the GPU: the one that takes the others'
    results may be the last to start, and the others have next to nothing to scan."""
    from minisglang_rdna4_b200.ops import cuda as K

    x = _rand(37, 16384, dtype=torch.float32)
    want = x.argmax(-1)
    busy = _rand(4096, 4096)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    got = []
    for _ in range(50):
        with torch.cuda.stream(side):
            busy = (busy @ busy).clamp(-1, 1)
        got += [K.argmax(x) for _ in range(8)]
    torch.cuda.synchronize()
    assert all(torch.equal(g.long(), want) for g in got)
