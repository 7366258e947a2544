"""The tcgen05 attention kernel over cache rows that are key and value, against float64."""
import pytest

pytestmark = pytest.mark.gpu


def _step(portions, rows, page=16):
    """A step's description for requests of (tokens, context), and one cache plane of `rows` numbers a row in shuffled pages."""
    import torch
    from kestrel_llm_b200.cache.manager import CacheManager
    from kestrel_llm_b200.engine import Entry, StepBatch
    from kestrel_llm_b200.parts.base import PagedKVSpec
    dev = torch.device("cuda:0")
    cache = CacheManager([PagedKVSpec(1, rows)], torch.bfloat16, dev, page, sum((n + c) // page + 2 for n, c in portions), len(portions), 4096)
    cache.shuffle_free(3)
    entries = []
    for i, (n, c) in enumerate(portions):
        cache.admit(i)
        cache.reserve(i, c)
        cache.commit(i, c)
        cache.reserve(i, n)
        entries.append(Entry(i, [1] * n))
    return cache, StepBatch(entries, cache, dev)


def _rows_of(cache, plane, i, length, page=16):
    """The first `length` rows of request i, in order."""
    import torch
    at = torch.tensor(cache.block_table(i, 0), device=plane.device)
    return plane[at].reshape(-1, plane.shape[-1])[:length]


@pytest.mark.parametrize("heads,portions", [(2, [(9, 1400)]), (16, [(40, 3000), (7, 90)])])
@pytest.mark.parametrize("rows,vd", [(72, 64), (256, 192)])         # values that a warp of the merge takes, and that a block takes
def test_a_gate_on_outputs_from_slices_is_rounded_with_them(heads, portions, rows, vd):
    """Queries of zero weigh all keys alike, and weights of one are exact in bfloat16: the output is a mean of values times the gate, rounded
    to bfloat16 once.  The float32 sums of up to 3,040 values around one are off by 2^-12 of the mean at most, a sixteenth of the rounding."""
    import torch
    from kestrel_llm_b200.csrc import ops
    torch.manual_seed(heads)
    cache, batch = _step(portions, rows)
    plane = cache.k[0]
    plane.normal_(1.0, 0.1)
    T = batch.num_tokens
    q, gate = torch.zeros(T, heads * rows, dtype=torch.bfloat16, device="cuda"), torch.rand(T, heads, device="cuda") + 0.25
    out = torch.full((T, heads * vd), float("nan"), dtype=torch.bfloat16, device="cuda")
    ops.attention_rows_tc(q, plane, out, batch, batch.block_table(0), 16, heads, 1, rows, vd, 0, rows ** -0.5, gate)
    assert ops.library().kestrel_attention_rows_tc_error() == 0
    want = torch.cat([_rows_of(cache, plane, i, n + c)[:, :vd].double().cumsum(0)[c:] / torch.arange(c + 1, c + n + 1, device="cuda")[:, None]
                      for i, (n, c) in enumerate(portions)])
    want = (want[:, None, :] * gate.double()[:, :, None]).reshape(T, -1)
    half = torch.exp2(torch.floor(torch.log2(want.abs())) - 8)
    assert ((out.double() - want).abs() / half).max().item() <= 1 + 1 / 16


@pytest.mark.parametrize("heads,portions", [(4, [(33, 100), (70, 0)]), (16, [(20, 1500), (9, 40)]), (1, [(300, 5), (1, 900)])])
@pytest.mark.parametrize("rows,vd", [(72, 64), (256, 192), (40, 24)])
@pytest.mark.parametrize("window", [0, 70])
def test_rows_against_float64_among_stale_pages(heads, portions, rows, vd, window):
    """Every number of the cache that no row may see is NaN, and one query row is infinite.  P is rounded to bfloat16, and so is the output:
    2^-8 of the weights' mean of |value| and 2^-8 of the output, beside 2^-12 of the largest for exp2 and float32 sums."""
    import torch
    from kestrel_llm_b200.csrc import ops
    torch.manual_seed(heads)
    cache, batch = _step(portions, rows)
    plane, dev, T = cache.k[0], "cuda", batch.num_tokens
    plane.fill_(float("nan"))
    kv = []
    for i, (n, c) in enumerate(portions):
        at = torch.arange(n + c, device=dev)
        seen = at[(at > c - window) | (window == 0)]
        x = torch.zeros(n + c, rows, dtype=torch.bfloat16, device=dev)
        x[seen] = torch.randn(len(seen), rows, device=dev).to(torch.bfloat16)
        plane[torch.tensor(cache.block_table(i, 0), device=dev)[seen // 16], 0, seen % 16] = x[seen]
        kv.append(x.double())
    q, gate = torch.randn(T, heads * rows, device=dev).to(torch.bfloat16), torch.rand(T, heads, device=dev)
    q[12, 7] = float("inf")                     # head 0 of one token
    out = torch.full((T, heads * vd), float("nan"), dtype=torch.bfloat16, device=dev)
    ops.attention_rows_tc(q, plane, out, batch, batch.block_table(0), 16, heads, 1, rows, vd, window, rows ** -0.5, gate)
    assert ops.library().kestrel_attention_rows_tc_error() == 0
    for i, (n, c) in enumerate(portions):
        t = slice(int(batch.cu_seqlens[i]), int(batch.cu_seqlens[i + 1]))
        s = torch.einsum("nhd,ld->hnl", q[t].view(n, heads, rows).double(), kv[i]) * rows ** -0.5
        dist = torch.arange(c, c + n, device=dev)[:, None] - torch.arange(n + c, device=dev)
        s = s.masked_fill((dist < 0) | ((dist >= window) & (window > 0)), -float("inf"))
        p = (s - s.amax(-1, keepdim=True)).exp()
        p = p / p.sum(-1, keepdim=True) * gate[t].double().t()[:, :, None]
        want, size = torch.einsum("hnl,ld->nhd", p, kv[i][:, :vd]), torch.einsum("hnl,ld->nhd", p, kv[i][:, :vd].abs())
        got = out[t].view(n, heads, vd).double()
        assert torch.equal(torch.isnan(want), torch.isnan(got))
        limit = 2.0 ** -8 * (size + want.abs()) + 2.0 ** -12 * want.nan_to_num().abs().max()
        assert ((got - want).abs() <= limit)[~torch.isnan(want)].all()
