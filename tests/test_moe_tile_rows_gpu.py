"""Grouped expert products on tcgen05: tiles that fetch and multiply no more than their own rows."""
import pytest

pytestmark = pytest.mark.gpu


# rows of every expert, and those that a tile fetches at a time: boxes of 32 up to 100 rows an expert on average, the last two sets on both sides of that
@pytest.mark.parametrize("counts,box", [((1, 15, 16, 17, 0, 31, 32, 33, 95, 96, 97, 127, 128, 129, 160, 225), 32), ((0, 1, 256, 255, 0, 3, 600), 128),
                                        ((0, 1, 256, 255, 17, 3, 900), 128), ((5, 33, 256, 255, 0, 3, 65, 111, 128, 144, 100), 32),
                                        ((5, 33, 256, 255, 0, 3, 65, 111, 128, 144, 101), 128)])
@pytest.mark.parametrize("K,ff", [(64, 136), (392, 72)])
@pytest.mark.parametrize("gated", [False, True])
def test_rows_of_every_tile_against_float64(counts, box, K, ff, gated):
    """One choice a token, so an expert's rows are as many as the tokens that name it.  The activation is rounded to bfloat16 between two
    products of float32 sums: 2^-8 of what the second product's terms add up to, and 2^-18 (64 roundings of 2^-24) of what the first's add
    up to through an activation of slope about one (the gated one: a product of two such)."""
    import torch
    from kestrel_llm_b200.csrc import ops
    torch.manual_seed(K)
    dev, E, T, N = "cuda", len(counts), sum(counts), 200
    ids = torch.repeat_interleave(torch.arange(E), torch.tensor(counts))[torch.randperm(T)].to(torch.int32)[:, None].to(dev)
    assert T >= ops.MOE_TC_MIN_PAIRS and ops.library().kestrel_moe_tc_box_rows(T, E) == box
    x = torch.randn(T, K, device=dev).to(torch.bfloat16)
    w1 = (torch.randn(E, (2 if gated else 1) * ff, K, device=dev) * K ** -0.5).to(torch.bfloat16)
    w2 = (torch.randn(E, N, ff, device=dev) * ff ** -0.5).to(torch.bfloat16)
    weights = torch.rand(T, 1, device=dev) + 0.5
    got = ops.moe_experts(x, ids, weights, w1, w2, None) if gated else ops.moe_experts_ungated(x, ids, weights, w1, w2, "silu")
    assert ops.library().kestrel_moe_tc_error() == 0
    for e in range(E):
        t = (ids[:, 0] == e).nonzero()[:, 0]
        h = x[t].double() @ w1[e].double().T
        size = x[t].double().abs() @ w1[e].double().abs().T
        a = torch.nn.functional.silu(h[:, :ff]) * (h[:, ff:] if gated else 1)
        off = 2.0 ** -8 * a.abs() + 2.0 ** -18 * size[:, :ff] * (h[:, ff:].abs() if gated else 1) + (2.0 ** -18 * size[:, ff:] * h[:, :ff].abs() if gated else 0)
        want, limit = a @ w2[e].double().T * weights[t], off @ w2[e].double().abs().T * weights[t]
        assert ((got[t].double() - want).abs() <= limit + 1e-6).all()
