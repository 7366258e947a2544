"""Products on CTA pairs with tiles of every width: an output is the same bits whatever tile it falls into."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.fixture
def tile():
    from kestrel_llm_b200.csrc import ops
    yield ops.gemm_tc_set_pair_tile
    ops.gemm_tc_set_pair_tile(0)


def _operands(T, N, K, seed=0):
    gen = torch.Generator(DEV).manual_seed(seed)
    return torch.randn((T, K), device=DEV, generator=gen).bfloat16(), torch.randn((N, K), device=DEV, generator=gen).bfloat16() * K ** -0.5


@pytest.mark.parametrize("T", [129, 176, 257, 700])                   # one tile and a row more, whole tiles of some widths, ragged
@pytest.mark.parametrize("N,K", [(256, 64), (264, 72), (1040, 1096)])  # fewer k-blocks than stages, ragged features and k-blocks
def test_slices_of_every_tile(tile, T, N, K):
    """bfloat16 products are exact in float32, so the error is that of the sums: 2^-24 K times the sum of magnitudes at the very most."""
    from kestrel_llm_b200.csrc import ops
    x, w = _operands(T, N, K)
    want = x.double() @ w.double().T
    bound = 2.0 ** -24 * (K + 1) * (x.double().abs() @ w.double().abs().T)
    for S in (1, 2):
        if S > 1 and K < 2048:
            continue
        first = None
        for columns in (256, 240, 224, 208, 192, 176, 160, 144, 128, 64, 16, 0):
            tile(columns)
            out = ops.gemm_tc(x, w, splits=S).data
            ops.raise_on_kernel_error()
            assert ((out.sum(0).double() - want).abs() <= bound).all(), f"tiles of {columns}"
            first = out if first is None else first
            assert torch.equal(out, first), f"tiles of {columns}"


@pytest.mark.parametrize("T,ff", [(129, 128), (300, 200), (700, 1552), (1030, 336)])
def test_gated_products_of_every_tile(tile, T, ff):
    """The SwiGLU product with tokens as the M operand: gate and up of half a tile's columns each."""
    from kestrel_llm_b200.csrc import ops
    K = 264
    x, w = _operands(T, 2 * ff, K, 1)
    g, u = (x.float() @ w.float().T).split(ff, 1)
    want = torch.nn.functional.silu(g) * u
    ops.library().kestrel_gemm_tc_set_swiglu_swapped(2)
    try:
        first = None
        for columns in (256, 224, 192, 160, 128, 64, 32, 0):
            tile(columns)
            out = torch.full((T, ff), float("nan"), dtype=torch.bfloat16, device=DEV)
            rc = ops.library().kestrel_gemm_tc_swiglu_w(x.data_ptr(), w.data_ptr(), out.data_ptr(), T, ff, K, K, K, ff, 1, ops._stream())
            ops.raise_on_kernel_error()
            # one rounding to bfloat16, and __expf in the sigmoid
            assert rc == 0 and ((out.float() - want).abs() <= 2.0 ** -8 * want.abs() + 1e-5).all(), f"tiles of {columns}"
            first = out if first is None else first
            assert torch.equal(out, first), f"tiles of {columns}"
    finally:
        ops.library().kestrel_gemm_tc_set_swiglu_swapped(1)


@pytest.mark.parametrize("T,N,K", [(2048, 2048, 136), (1800, 2056, 72), (2500, 1032, 264)])     # uncut: as many tiles as fill the pairs; ragged ends
def test_added_to_the_stream_by_every_tile(tile, T, N, K):
    """The product added in place: float32 sums of exact products and one more addition, whatever the tile."""
    from kestrel_llm_b200.csrc import ops
    x, w = _operands(T, N, K, 3)
    held = torch.randn((T, N), device=DEV, generator=torch.Generator(DEV).manual_seed(4)) * 8
    want = held.double() + x.double() @ w.double().T
    bound = 2.0 ** -24 * (K + 2) * (x.double().abs() @ w.double().abs().T + held.double().abs())
    taken = 0
    for columns in (256, 240, 208, 176, 128, 16, 0):
        tile(columns)
        out = held.clone()
        rc = ops.library().kestrel_gemm_tc_add(x.data_ptr(), w.data_ptr(), out.data_ptr(), T, N, K, K, K, N, ops._stream())
        ops.raise_on_kernel_error()
        taken += rc == 0
        assert rc == 1 or ((out.double() - want).abs() <= bound).all(), f"tiles of {columns}"
        assert rc == 0 or torch.equal(out, held)
    assert taken


def test_a_tile_is_chosen_by_its_rounds():
    """1,024 tokens of 3,072 features: 48 tiles of 256 leave a third of 74 pairs idle; the tile taken fills them better, and sums are
    cut along K no more than before."""
    from kestrel_llm_b200.csrc import ops
    x, w = _operands(1024, 3072, 2048, 2)
    out = ops.gemm_tc(x, w).data
    want = x.float() @ w.float().T
    ops.raise_on_kernel_error()
    assert torch.allclose(out.sum(0), want, rtol=0, atol=2.0 ** -20 * float(want.abs().max()) * 64)
