"""Attention kernels that find their tiles in the step's cumulative lengths instead of reading lists that the host made."""
import pytest

pytestmark = pytest.mark.gpu


def _step(counts, heads, dim, contexts):
    import torch
    from kestrel_llm_b200.cache.manager import CacheManager
    from kestrel_llm_b200.engine import Entry, StepBatch
    from kestrel_llm_b200.parts.base import PagedKVSpec
    dev = torch.device("cuda:0")
    cache = CacheManager([PagedKVSpec(heads, dim)], torch.bfloat16, dev, 16, sum((n + c) // 16 + 2 for n, c in zip(counts, contexts)), len(counts), 4096)
    cache.shuffle_free(5)
    cache.k[0].normal_()
    cache.v[0].normal_()
    entries = []
    for i, (n, c) in enumerate(zip(counts, contexts)):
        cache.admit(i)
        cache.reserve(i, c)
        cache.commit(i, c)
        cache.reserve(i, n)
        entries.append(Entry(i, [1] * n))
    return cache, StepBatch(entries, cache, dev)


# one request, tiles that end with a request and one row behind it, requests of one token on both sides of a warp's 32, many tiles of one
STEPS = [[1], [32], [33, 1, 64], [1] * 31 + [50], [1] * 32 + [50], [1] * 70 + [33] + [2] * 30, [300, 1, 1, 129]]


@pytest.mark.parametrize("counts", STEPS)
@pytest.mark.parametrize("rows", [128, 256])
@pytest.mark.parametrize("H,G", [(8, 2), (3, 3)])
def test_found_tiles_are_the_listed_ones(counts, rows, H, G):
    import torch
    from kestrel_llm_b200.csrc import ops
    torch.manual_seed(H)
    contexts = [(37 * i) % 200 for i in range(len(counts))]
    cache, batch = _step(counts, G, 128, contexts)
    T = batch.num_tokens
    q, gate = torch.randn(T, H * 128, device="cuda").to(torch.bfloat16), torch.rand(T, H, device="cuda")
    got = []
    for seq, row0 in (ops.row_tiles(batch, H // G, rows), (None, None)):
        out = torch.full_like(q, float("nan"))
        ops.attention_tc(q, cache.k[0], cache.v[0], out, seq, row0, batch.cu_seqlens, batch.kv_lens, batch.block_table(0), 16, H, G, 128, 60,
                         128 ** -0.5, rows_per_tile=rows, keep_first=5, gate=gate, tiles=ops.count_row_tiles(batch, H // G, rows))
        got.append(out)
    assert ops.attention_tc_error() == 0
    assert torch.equal(*got) and not torch.isnan(got[0]).any()


@pytest.mark.parametrize("counts", STEPS)
@pytest.mark.parametrize("longest", [0, 2500])          # in one slice of keys, and in several that a second kernel merges
def test_rows_in_found_tiles_do_not_depend_on_the_step(counts, longest):
    """Every request's outputs over cache rows are those of the request in a step of its own, up to the two roundings to bfloat16 (of P and of
    the output, 2^-8 each of the largest) that key ranges cut elsewhere may move."""
    import torch
    from kestrel_llm_b200.csrc import ops
    torch.manual_seed(len(counts))
    contexts = [(37 * i) % 200 for i in range(len(counts))]
    contexts[-1] += longest
    cache, batch = _step(counts, 1, 72, contexts)
    plane, heads = cache.k[0], 4
    q = torch.randn(batch.num_tokens, heads * 72, device="cuda").to(torch.bfloat16)

    def run(q, b):
        out = torch.full((q.shape[0], heads * 64), float("nan"), dtype=torch.bfloat16, device="cuda")
        ops.attention_rows_tc(q, plane, out, b, b.block_table(0), 16, heads, 1, 72, 64, 0, 72 ** -0.5)
        return out
    whole = run(q, batch)
    assert not torch.isnan(whole).any()
    from kestrel_llm_b200.engine import Entry, StepBatch
    for i in {0, len(counts) // 2, len(counts) - 1}:
        t = slice(batch.cu_seqlens_host[i], batch.cu_seqlens_host[i + 1])
        alone = run(q[t].contiguous(), StepBatch([Entry(i, [1] * counts[i])], cache, torch.device("cuda:0")))
        assert (alone.float() - whole[t].float()).abs().max() <= 2.0 ** -7 * alone.float().abs().max()
    assert ops.library().kestrel_attention_rows_tc_error() == 0


def test_layers_make_no_lists(monkeypatch):
    """A step of a layer with kept tokens and a gate, and of one over cached latents behind a context, takes no list of tiles from the host."""
    import torch
    from kestrel_llm_b200.cache.manager import CacheManager
    from kestrel_llm_b200.csrc import ops
    from kestrel_llm_b200.engine import Entry, StepBatch
    from kestrel_llm_b200.parts import GatedWindowAttention, LatentAttention

    def listed(*a, **kw):
        raise AssertionError("a list of tiles was made")
    monkeypatch.setattr(ops, "row_tiles", listed)
    dev, bf16 = torch.device("cuda:0"), torch.bfloat16
    for mixer in (GatedWindowAttention(256, 8, 2, 128, 128, bf16, dev, "m.", 128 ** -0.5, 1e-6, window=64, keep_first=4),
                  LatentAttention(256, 4, 32, 32, 64, 64, bf16, dev, "m.", 32 ** -0.5, 1e-6)):
        for slot in mixer.weight_slots():
            slot.dest.normal_(0.0, 0.05)
        cache = CacheManager([mixer.cache_spec()], bf16, dev, 16, 40, 1, 512)
        cache.k[0].zero_()
        cache.admit(0)
        cache.reserve(0, 100)
        cache.commit(0, 100)
        cache.reserve(0, 90)
        batch = StepBatch([Entry(0, [1] * 90)], cache, dev)
        x = torch.randn(90, 256, device=dev).to(bf16)
        mixer.forward(x, batch, cache.layer(0))
    ops.raise_on_kernel_error()
