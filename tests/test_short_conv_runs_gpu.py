"""Short convolutions over time: runs of tokens that end in a request or at the step's end, filters on and off 16-byte boundaries."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("counts", [(511,), (512,), (513, 1, 2, 3), (7, 0, 600, 5), (3,) * 171])
@pytest.mark.parametrize("taps", [1, 2, 3, 4, 5, 9])
@pytest.mark.parametrize("channels", [20, 516, 37])
def test_convolutions_against_float64(counts, taps, channels):
    """`taps` multiply-adds, a bias and a silu of slope at most 1.1: taps + 4 roundings of 2^-24 of what the terms add up to, and silu's own
    few.  An aligned and an unaligned copy of the filter leave the same bits, in the outputs and in the kept inputs."""
    import torch
    from types import SimpleNamespace
    from kestrel_llm_b200.csrc import ops
    torch.manual_seed(taps)
    dev, n, T = "cuda", len(counts), sum(counts)
    cu = torch.tensor([0, *counts]).cumsum(0).to(torch.int32).to(dev)
    seq = torch.repeat_interleave(torch.arange(n), torch.tensor(counts)).to(torch.int32).to(dev)
    slots = torch.randperm(n).to(torch.int32).to(dev)
    batch = SimpleNamespace(seq_of_token=seq, cu_seqlens=cu, slots=slots, num_seqs=n)
    col0 = 4
    p = torch.randn(2, T, channels + 8, device=dev)
    room = torch.randn(taps * channels + 1, device=dev)
    bias = torch.randn(channels, device=dev)
    before = torch.randn(n, (taps - 1) * channels + 4, device=dev)
    got = []
    for off in (0, 1):
        w = torch.empty_like(room)[off:off + taps * channels].view(taps, channels).copy_(room[:taps * channels].view(taps, channels))
        out, state = torch.full((T, channels), float("nan"), device=dev), before.clone()
        x = ops.Partials(p)
        ops.short_conv(x, w, bias, state, 4, batch, out, col0)
        got.append((out, state))
    assert torch.equal(got[0][0], got[1][0]) and torch.equal(got[0][1], got[1][1])
    u, w64 = (p[0] + p[1])[:, col0:col0 + channels].double(), room[:taps * channels].view(taps, channels).double()
    for i, c in enumerate(counts):
        tail = before[slots[i].long(), 4:].view(taps - 1, channels).double()
        full = torch.cat([tail, u[int(cu[i]):int(cu[i]) + c]])
        terms = torch.stack([full[j:j + c] * w64[j] for j in range(taps)]).view(taps, c, channels)
        z, size = terms.sum(0) + bias.double(), terms.abs().sum(0) + bias.double().abs()
        want = torch.nn.functional.silu(z)
        assert ((got[0][0][int(cu[i]):int(cu[i]) + c].double() - want).abs() <= 2.0 ** -24 * ((taps + 4) * 1.1 * size + 16 * want.abs())).all()
        assert torch.equal(got[0][1][slots[i].long(), 4:].view(taps - 1, channels).double(), full[c:])
