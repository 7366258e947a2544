"""The tcgen05 attention kernel with one row tile a CTA, whose key tiles two streams take in turn, against two row tiles a CTA."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H,G", [(4, 4), (8, 2), (3, 1)])
@pytest.mark.parametrize("portions", [[(1, 0), (40, 0)], [(128, 0)], [(70, 90), (33, 223)], [(5, 380), (129, 100), (64, 1000)], [(3, 0), (70, 500)]])
@pytest.mark.parametrize("kind", ["plain", "window", "sink", "cap", "rel", "kept", "sliced", "sliced sink"])
def test_key_tiles_in_two_streams(H, G, portions, kind):
    """One, two and more key tiles, rows that end in either stream's tile, rows that see nothing of a slice.  Both forms round P to bfloat16
    (2^-9 of a weight) against references that differ, and the output: twice 2^-8 of the largest value and a half."""
    import torch
    from kestrel_llm_b200.cache.manager import CacheManager
    from kestrel_llm_b200.csrc import ops
    from kestrel_llm_b200.engine import Entry, StepBatch
    from kestrel_llm_b200.parts.base import PagedKVSpec
    torch.manual_seed(H)
    dev, page = torch.device("cuda:0"), 16
    cache = CacheManager([PagedKVSpec(G, 128)], torch.bfloat16, dev, page, sum((n + c) // page + 2 for n, c in portions), len(portions), 2048)
    cache.shuffle_free(3)
    cache.k[0].normal_()
    cache.v[0].normal_()
    entries = []
    for i, (n, c) in enumerate(portions):
        cache.admit(i)
        cache.reserve(i, c)
        cache.commit(i, c)
        cache.reserve(i, n)
        entries.append(Entry(i, [1] * n))
    batch = StepBatch(entries, cache, dev)
    T = batch.num_tokens
    q = torch.randn(T, H * 128, device=dev).to(torch.bfloat16)
    opts, window = {}, 100 if kind in ("window", "kept") else 0
    sink = torch.randn(H, device=dev)
    if kind in ("sink", "sliced sink"):
        opts["score"] = ops.ScoreOptions(0.0, None, None, None, "softmax_sink", sink, None, None)
    elif kind == "cap":
        opts["score"] = ops.ScoreOptions(2.0, None, None, None, "softmax", None, None, None)
    elif kind == "rel":
        bucket = torch.arange(200, dtype=torch.int32, device=dev) // 30
        opts["score"] = ops.ScoreOptions(0.0, None, None, None, "softmax", None, torch.randn(7, H, device=dev), bucket)
    elif kind == "kept":
        opts.update(keep_first=5, gate=torch.rand(T, H, device=dev))
    if kind.startswith("sliced"):
        opts.update(slices=-(-batch.max_kv_len // 256), slice_len=256)
    got = []
    for rows in (256, 128):
        out = torch.full_like(q, float("nan"))
        seq, row0 = ops.row_tiles(batch, H // G, rows)
        ops.attention_tc(q, cache.k[0], cache.v[0], out, seq, row0, batch.cu_seqlens, batch.kv_lens, batch.block_table(0), page, H, G, 128, window,
                         128 ** -0.5, rows_per_tile=rows, **opts)
        got.append(out.float())
    assert ops.attention_tc_error() == 0
    assert (got[0] - got[1]).abs().max() <= 2.0 ** -7 * got[0].abs().max() * 1.5


def test_rows_of_a_tile_follow_the_step():
    """Tiles of 128 while they fit the SMs or where one request's last tokens set the pace, of 256 for many portions and long prompts."""
    from types import SimpleNamespace
    from kestrel_llm_b200.csrc import ops

    def rows(portions, group, nkv, window=0, keep=0):
        import torch
        b = SimpleNamespace(counts=[n for n, _ in portions], starts=[s for _, s in portions], device_buffer=torch.empty(1, device="cuda"))
        return ops.attention_tc_tiles(b, group, nkv, window, keep)[2]
    assert rows([(500, 750)], 4, 8) == 128 and rows([(2048, 0)], 4, 4) == 128
    assert rows([(500, 0)] * 4, 4, 4) == 256 and rows([(2048, 0)], 4, 8) == 256 and rows([(2048, 0)], 4, 4, 1024, 4) == 256


@pytest.mark.parametrize("H,G", [(4, 4), (8, 2), (3, 1)])
@pytest.mark.parametrize("portions", [[(1, 0), (140, 0)], [(70, 90), (33, 223)], [(129, 100), (64, 1000)]])
@pytest.mark.parametrize("rows", [128, 256])
@pytest.mark.parametrize("kind", ["plain", "window", "sink", "cap", "rel", "kept", "sliced", "sliced sink"])
def test_streams_against_float64_among_stale_pages(H, G, portions, rows, kind):
    """Every number of the cache that no row may see is NaN, and one query row is infinite.  P is rounded to bfloat16, and so is the output:
    2^-8 of the weights' mean of |v| and 2^-8 of the output, beside 2^-12 of the largest for exp2, the caps and float32 sums."""
    import torch
    from kestrel_llm_b200.cache.manager import CacheManager
    from kestrel_llm_b200.csrc import ops
    from kestrel_llm_b200.engine import Entry, StepBatch
    from kestrel_llm_b200.parts.base import PagedKVSpec
    torch.manual_seed(H)
    dev, page, window, keep = torch.device("cuda:0"), 16, 100 if kind in ("window", "kept") else 0, 5 if kind == "kept" else 0
    cache = CacheManager([PagedKVSpec(G, 128)], torch.bfloat16, dev, page, sum((n + c) // page + 2 for n, c in portions), len(portions), 2048)
    cache.shuffle_free(3)
    cache.k[0].fill_(float("nan"))
    cache.v[0].fill_(float("nan"))
    entries, kv = [], []
    for i, (n, c) in enumerate(portions):
        cache.admit(i)
        cache.reserve(i, c)
        cache.commit(i, c)
        cache.reserve(i, n)
        entries.append(Entry(i, [1] * n))
        at = torch.arange(n + c, device=dev)
        seen = at[(at < keep) | (at > c - window) | (window == 0)]
        where = torch.tensor(cache.block_table(i, 0), device=dev)[seen // page], seen % page
        kv.append([])
        for plane in (cache.k[0], cache.v[0]):
            x = torch.zeros(n + c, G, 128, dtype=torch.bfloat16, device=dev)
            x[seen] = torch.randn(len(seen), G, 128, device=dev).to(torch.bfloat16)
            plane[where[0], :, where[1]] = x[seen]
            kv[-1].append(x.double())
    batch = StepBatch(entries, cache, dev)
    T = batch.num_tokens
    q = torch.randn(T, H * 128, device=dev).to(torch.bfloat16)
    if T > 130:
        q[T - 70, 7] = float("inf")             # head 0 of one token
    sink, bucket = torch.randn(H, device=dev), torch.arange(200, dtype=torch.int32, device=dev) // 30
    rel, gate, opts = torch.randn(7, H, device=dev), torch.rand(T, H, device=dev), {}
    if kind in ("sink", "sliced sink"):
        opts["score"] = ops.ScoreOptions(0.0, None, None, None, "softmax_sink", sink, None, None)
    elif kind == "cap":
        opts["score"] = ops.ScoreOptions(2.0, None, None, None, "softmax", None, None, None)
    elif kind == "rel":
        opts["score"] = ops.ScoreOptions(0.0, None, None, None, "softmax", None, rel, bucket)
    elif kind == "kept":
        opts.update(keep_first=keep, gate=gate)
    if kind.startswith("sliced"):
        opts.update(slices=-(-batch.max_kv_len // 256), slice_len=256)
    out = torch.full_like(q, float("nan"))
    seq, row0 = ops.row_tiles(batch, H // G, rows)
    ops.attention_tc(q, cache.k[0], cache.v[0], out, seq, row0, batch.cu_seqlens, batch.kv_lens, batch.block_table(0), page, H, G, 128, window,
                     128 ** -0.5, rows_per_tile=rows, **opts)
    assert ops.attention_tc_error() == 0
    for i, (n, c) in enumerate(portions):
        t = slice(int(batch.cu_seqlens[i]), int(batch.cu_seqlens[i + 1]))
        k, v = (x.repeat_interleave(H // G, dim=1) for x in kv[i])
        s = torch.einsum("nhd,lhd->hnl", q[t].view(n, H, 128).double(), k) * 128 ** -0.5
        dist = torch.arange(c, c + n, device=dev)[:, None] - torch.arange(n + c, device=dev)
        if kind == "cap":
            s = 2.0 * torch.tanh(s / 2.0)
        if kind == "rel":
            s = s + rel[bucket[dist.clamp(0, 199)].long()].permute(2, 0, 1).double()
        hidden = dist < 0
        if window:
            hidden = hidden | ((dist >= window) & (torch.arange(n + c, device=dev) >= keep))
        s = s.masked_fill(hidden, -float("inf"))
        top = s.amax(-1, keepdim=True)
        p = (s - top).exp()
        total = p.sum(-1, keepdim=True) + ((sink.double()[:, None, None] - top).exp() if "sink" in kind else 0.0)
        p = p / total
        if kind == "kept":
            p = p * gate[t].double().t()[:, :, None]
        want, size = torch.einsum("hnl,lhd->nhd", p, v), torch.einsum("hnl,lhd->nhd", p, v.abs())
        got = out[t].view(n, H, 128).double()
        assert torch.equal(torch.isnan(want), torch.isnan(got))
        limit = 2.0 ** -8 * (size + want.abs()) + 2.0 ** -12 * want.nan_to_num().abs().max()
        assert ((got - want).abs() <= limit)[~torch.isnan(want)].all()
