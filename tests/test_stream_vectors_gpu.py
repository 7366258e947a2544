"""Kernels of the residual stream in vectors: widths that are whole vectors and widths that are not, tensors on any boundary."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _shifted(t, by):
    """The same numbers ``by`` elements behind a 16-byte boundary."""
    flat = torch.empty(t.numel() + 16, dtype=t.dtype, device=DEV)
    out = flat[by:by + t.numel()].view(t.shape)
    return out.copy_(t)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("d", [1, 4, 8, 12, 2040, 2048, 2056, 8200])
@pytest.mark.parametrize("T,shift", [(1, 0), (33, 0), (33, 2)])
def test_embedding_rows(dtype, d, T, shift):
    from kestrel_llm_b200.csrc import ops
    gen = torch.Generator(DEV).manual_seed(d)
    table = _shifted(torch.randn((50, d), device=DEV, generator=gen).to(dtype), shift)
    ids = torch.randint(0, 50, (T,), device=DEV, generator=gen, dtype=torch.int32)
    out = torch.full((T, d), float("nan"), device=DEV)
    ops.embed(table, ids, out)
    assert torch.equal(out, table[ids.long()].float())


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("S", [1, 2, 3, 4, 5, 9])
@pytest.mark.parametrize("T,width,shift", [(1, 4, 0), (7, 1024, 0), (33, 1028, 0), (33, 1030, 0), (9, 260, 1)])
@pytest.mark.parametrize("bias", [False, True])
def test_slices_into_a_tensor(dtype, S, T, width, shift, bias):
    """Slices are added in ascending order, the bias last: the same bits as the sums one by one."""
    from kestrel_llm_b200.csrc import ops
    gen = torch.Generator(DEV).manual_seed(width + S)
    parts = _shifted(torch.randn((S, T, width), device=DEV, generator=gen), shift)
    b = torch.randn(width, device=DEV, generator=gen) if bias else None
    want = torch.zeros((T, width), device=DEV)
    for s in range(S):
        want = want + parts[s]
    if bias:
        want = want + b
    out = ops.Partials(parts, b).reduce(dtype)
    assert torch.equal(out, want.to(dtype))


@pytest.mark.parametrize("d", [4, 60, 250, 2048, 2052, 4100, 11996, 11999])
@pytest.mark.parametrize("Sa,Sb", [(1, 1), (2, 9)])
def test_two_results_normed_and_combined(d, Sa, Sb):
    """Against float64 (float32 sums of d squares and of slices: 2^-20 of the largest is four roundings and more), and every row the same bits
    among many rows and alone."""
    from kestrel_llm_b200.csrc import ops
    gen = torch.Generator(DEV).manual_seed(d)
    T = 300
    a, b = (torch.randn((S, T, d), device=DEV, generator=gen) for S in (Sa, Sb))
    wa, wb = (torch.randn(d, device=DEV, generator=gen) for _ in range(2))
    got = ops.combine_normed(ops.Partials(a), wa, ops.Partials(b), wb, 1e-6, 0.5).data[0]
    alone = ops.combine_normed(ops.Partials(a[:, 7:8].contiguous()), wa, ops.Partials(b[:, 7:8].contiguous()), wb, 1e-6, 0.5).data[0]
    x, y = a.double().sum(0), b.double().sum(0)
    want = 0.5 * (x / torch.sqrt((x * x).mean(1, keepdim=True) + 1e-6) * wa + y / torch.sqrt((y * y).mean(1, keepdim=True) + 1e-6) * wb)
    assert ((got - want).abs() <= 2.0 ** -20 * want.abs().max()).all()
    assert torch.equal(got[7], alone[0])
