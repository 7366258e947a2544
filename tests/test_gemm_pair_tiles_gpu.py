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


# T: one tile and a row more, whole tiles of some widths, ragged.  N, K: fewer k-blocks than stages, ragged features and k-blocks, slices that refill
# the ring, with a last one that is shorter; the last size has more tiles than pairs
@pytest.mark.parametrize("T,N,K", [(T, N, K) for T in (129, 176, 257, 700) for N, K in ((256, 64), (264, 72), (1040, 1096), (520, 2056), (264, 3080))] + [(2100, 2568, 1096)])
def test_slices_of_every_tile(tile, T, N, K):
    """bfloat16 products are exact in float32, so the error is that of the sums: 2^-24 K times the sum of magnitudes at the very most.  Weights
    that are fetched before the kernel before ends are the same ones."""
    from kestrel_llm_b200.csrc import ops
    x, w = _operands(T, N, K)
    want = x.double() @ w.double().T
    bound = 2.0 ** -24 * (K + 1) * (x.double().abs() @ w.double().abs().T)
    blocks, cut = -(-K // 64), 0
    for S in (1, 2, 3):
        if -(-blocks // S) * (S - 1) >= blocks:         # a slice would be empty
            continue
        first = None
        for columns in (256, 240, 224, 208, 192, 176, 160, 144, 128, 64, 16, 0):
            tile(columns)
            for static in (False, True):
                out = ops.gemm_tc(x, w, splits=S, weights_static=static).data
                assert out.shape[0] == S
                ops.raise_on_kernel_error()
                assert ((out.sum(0).double() - want).abs() <= bound).all(), f"tiles of {columns}, {S} slices"
                first = out if first is None else first
                assert torch.equal(out, first), f"tiles of {columns}, {S} slices"
        cut += S > 1
    assert cut == (0 if K <= 64 else 1 if K <= 128 else 2)


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
    """1,024 tokens of 3,072 features: 48 tiles of 256 leave a third of 74 pairs idle; the tile taken fills them better in as many rounds, and
    the sums are not cut along K."""
    from kestrel_llm_b200.csrc import ops
    T, N, K = 1024, 3072, 2048
    x, w = _operands(T, N, K, 2)
    out = ops.gemm_tc(x, w).data
    want = x.float() @ w.float().T
    ops.raise_on_kernel_error()
    columns, pairs = ops.library().kestrel_gemm_tc_pair_columns(T, N, K, 1), torch.cuda.get_device_properties(0).multi_processor_count // 2
    assert out.shape[0] == 1 and -(-T // 256) * 12 < -(-T // columns) * 12 <= pairs
    assert torch.allclose(out.sum(0), want, rtol=0, atol=2.0 ** -20 * float(want.abs().max()) * 64)
