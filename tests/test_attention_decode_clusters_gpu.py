"""Decode attention whose slices are merged by clusters where every one is resident, else through scratch."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("hd", [64, 128])
@pytest.mark.parametrize("requests", [1, 8, 9, 12, 18, 19])
@pytest.mark.parametrize("capped", [False, True])
def test_slices_by_clusters_against_float64(hd, requests, capped):
    """Sums are float32 of bfloat16 products and P is rounded to bfloat16, and so is the output: 2^-8 of the weights' mean of |value| and 2^-8
    of the output, beside 2^-12 of the largest for exp2 and float32 sums (a cap of scores by 50 in float32 moves them by less)."""
    import torch
    from kestrel_llm_b200.cache.manager import CacheManager
    from kestrel_llm_b200.csrc import ops
    from kestrel_llm_b200.engine import Entry, StepBatch
    from kestrel_llm_b200.parts.base import PagedKVSpec
    torch.manual_seed(requests)
    dev, page, nq, nkv = torch.device("cuda:0"), 16, 16, 8
    contexts = [1100 - 37 * i for i in range(requests)]
    cache = CacheManager([PagedKVSpec(nkv, hd)], torch.bfloat16, dev, page, sum(c // page + 2 for c in contexts), requests, 2048)
    cache.shuffle_free(3)
    entries = []
    for i, c in enumerate(contexts):
        cache.admit(i)
        cache.reserve(i, c)
        cache.commit(i, c)
        cache.reserve(i, 1)
        entries.append(Entry(i, [1]))
    batch = StepBatch(entries, cache, dev)
    k, v = cache.k[0].normal_(), cache.v[0].normal_()
    q = torch.randn(requests, nq * hd, device=dev).to(torch.bfloat16)
    out = torch.full_like(q, float("nan"))
    if capped:
        assert ops.attention_decode_capped(q, k, v, batch, batch.block_table(0), page, out, nq, nkv, hd, 0, hd ** -0.5, 50.0)
    else:
        ops.attention(ops.AttentionPlanner(requests, requests), q, k, v, batch, 0, page, out, nq, nkv, hd, 0, hd ** -0.5)
    assert ops.attention_decode_error() == 0
    lib = ops.library()
    most = lib.kestrel_attention_decode_cluster_slices()
    held = [lib.kestrel_attention_decode_slots(hd)] * 2 + [lib.kestrel_attention_decode_clusters(hd, s) for s in range(2, most + 1)]
    assert all(1 <= held[s] * s <= held[0] for s in range(2, most + 1))
    # as many slices as let every CTA be resident, and clusters of them only where every one is
    ctas, keys = requests * nkv, contexts[0] + 1
    slices = ops.decode_capped_slices(hd, ctas, keys) if capped else lib.kestrel_attention_slices(1, hd, ctas, keys)
    assert slices == max(1, min(held[0] // ctas, -(-keys // 128), most if capped else 32))
    for s in range(1, most + 2):
        assert lib.kestrel_attention_slices_in_clusters(hd, ctas, s) == (1 < s <= most and ctas <= held[s])
    for i, c in enumerate(contexts):
        at = torch.tensor(cache.block_table(i, 0), device=dev)
        rows = [x[at].transpose(0, 1).reshape(nkv, -1, hd)[:, :c + 1].double().repeat_interleave(nq // nkv, 0) for x in (k, v)]
        s = torch.einsum("hd,hld->hl", q[i].view(nq, hd).double(), rows[0]) * hd ** -0.5
        p = (50 * torch.tanh(s / 50) if capped else s).softmax(-1)
        want, size = torch.einsum("hl,hld->hd", p, rows[1]), torch.einsum("hl,hld->hd", p, rows[1].abs())
        limit = 2.0 ** -8 * (size + want.abs()) + 2.0 ** -12 * want.abs().max()
        assert ((out[i].view(nq, hd).double() - want).abs() <= limit).all()


@pytest.mark.parametrize("hd,nq,nkv", [(64, 16, 8), (128, 24, 3), (128, 32, 2)])
@pytest.mark.parametrize("slices", [2, 3, 4])
def test_scratch_and_clusters_give_the_same_bits(hd, nq, nkv, slices):
    """Requests of one to 1,100 keys, so that some have fewer keys than slices reach: the same parts merged in the same order."""
    import torch
    from kestrel_llm_b200.cache.manager import CacheManager
    from kestrel_llm_b200.csrc import ops
    from kestrel_llm_b200.engine import Entry, StepBatch
    from kestrel_llm_b200.parts.base import PagedKVSpec
    torch.manual_seed(slices)
    dev, page, contexts = torch.device("cuda:0"), 16, [1099, 0, 63, 700, 256, 1000]
    cache = CacheManager([PagedKVSpec(nkv, hd)], torch.bfloat16, dev, page, sum(c // page + 2 for c in contexts), len(contexts), 2048)
    entries = []
    for i, c in enumerate(contexts):
        cache.admit(i)
        cache.reserve(i, c)
        cache.commit(i, c)
        cache.reserve(i, 1)
        entries.append(Entry(i, [1]))
    batch, n = StepBatch(entries, cache, dev), len(contexts)
    k, v = cache.k[0].normal_(), cache.v[0].normal_()
    q = torch.randn(n, nq * hd, device=dev).to(torch.bfloat16)
    table, rows, first = batch.block_table(0), torch.arange(n, dtype=torch.int32, device=dev), torch.zeros(n, dtype=torch.int32, device=dev)
    got = []
    for scratch in (False, True):
        out = torch.full_like(q, float("nan"))
        part = torch.full((n * nq * slices * (hd + 2),), float("nan"), device=dev) if scratch else None
        ops._check(ops.library().kestrel_attention_decode(
            q.data_ptr(), k.data_ptr(), v.data_ptr(), out.data_ptr(), part.data_ptr() if scratch else None, part.data_ptr() + 4 * n * nq * slices * hd if scratch else None,
            rows.data_ptr(), first.data_ptr(), n, batch.cu_seqlens.data_ptr(), batch.kv_lens.data_ptr(), table.data_ptr(), table.shape[1], table.stride(0), page,
            int(k.shape[0]), n, nq, nkv, hd, 0, slices, -(-1100 // (64 * slices)) * 64, None, hd ** -0.5, ops._stream()))
        got.append(out)
    assert ops.attention_decode_error() == 0 and torch.isfinite(got[0].float()).all() and torch.equal(got[0], got[1])
