"""The vector form of the kernel between a fused product and attention (bfloat16) against the general one (float32 storage)."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nq,nkv,hd", [(4, 2, 32), (16, 4, 128), (6, 3, 64), (1, 1, 128), (0, 5, 128)])
@pytest.mark.parametrize("T,S", [(1, 3), (5, 1), (33, 2)])
@pytest.mark.parametrize("rot,pairing", [(0, ""), (32, "interleaved"), (10, "interleaved"), (16, "half"), (32, "half")])
@pytest.mark.parametrize("qk_norm,weights,v_norm,bias,temp,gate,has_kv", [
    ("head", True, False, False, None, True, True), (None, False, True, True, None, False, True), ("head", False, False, True, (0.3, 4), False, False)])
def test_vector_form_against_the_general_kernel(nq, nkv, hd, T, S, rot, pairing, qk_norm, weights, v_norm, bias, temp, gate, has_kv):
    """Both work in float32; they differ by the order of a sum of squares of a head (a few 2^-24 of a value) and then by the storage type: a
    bfloat16 has eight significant bits, so rounding to it moves a value by at most half of its last place, 2^-8 of it."""
    import torch
    from kestrel_llm_b200.csrc import ops
    from kestrel_llm_b200.parts.base import Rotation
    if nq == 0 and not has_kv:
        pytest.skip("nothing to prepare")
    torch.manual_seed(hd + T)
    page, dev = 16, "cuda"
    cols = nq * hd + (2 * nkv * hd if has_kv else 0) + (nq if gate else 0)
    cols += -cols % 4
    data = torch.randn(S, T, cols, device=dev)
    b = torch.randn(cols, device=dev) if bias else None
    pos = (torch.randperm(60)[:T] if T <= 60 else torch.arange(T)).to(torch.int32).to(dev)
    seq = torch.zeros(T, dtype=torch.int32, device=dev)
    table = torch.randperm(4, dtype=torch.int32, device=dev)[None].contiguous()
    qw, kw = (torch.rand(hd, device=dev) + 0.5 for _ in range(2)) if weights else (None, None)
    rotation = Rotation(torch.rand(rot // 2, device=dev), rot, pairing, 1.2) if rot else None
    got = []
    for dtype in (torch.float32, torch.bfloat16):
        k, v = (torch.zeros(4, nkv, page, hd, dtype=dtype, device=dev) for _ in range(2))
        q = torch.zeros(T, nq * hd, dtype=dtype, device=dev)
        g = torch.zeros(T, nq, device=dev) if gate else None
        ops.attn_prepare_ex(ops.Partials(data.clone(), b), qw, kw, qk_norm, 1e-6, pos, seq, table, page, k, v, q, g, nq, nkv, hd, hd, has_kv,
                            v_norm=v_norm, rotation=rotation, q_temp=temp)
        got.append([q.float(), k.float(), v.float()] + ([g] if gate else []))
    for a, c in zip(*got):
        if a.numel():
            assert (a - c).abs().le((2.0 ** -8 + 2.0 ** -21) * a.abs() + 1e-6).all()


@pytest.mark.parametrize("H,dv", [(16, 128), (5, 64), (3, 32), (1, 128), (9, 32)])
@pytest.mark.parametrize("T,S", [(1, 2), (37, 1), (513, 3)])
@pytest.mark.parametrize("gate,per_channel", [(True, True), (True, False), (False, False)])
def test_head_norm_in_vectors(H, dv, T, S, gate, per_channel):
    """bfloat16 results of the read-outs' norm and gate against the float32 ones: a rounding to eight bits, and the order of a sum of squares."""
    import torch
    from kestrel_llm_b200.csrc import ops
    torch.manual_seed(T)
    o = torch.randn(T, H * dv, device="cuda")
    w = torch.rand(H * dv if per_channel else dv, device="cuda") + 0.5
    g = ops.Partials(torch.randn(S, T, H * dv + 8, device="cuda")) if gate else None
    exact, got = torch.empty(T, H * dv, device="cuda"), torch.empty(T, H * dv, dtype=torch.bfloat16, device="cuda")
    for out in (exact, got):
        ops.head_norm_gate(o, w, 1e-6, g, 4 if gate else 0, out, H, dv)
    assert (exact - got.float()).abs().le((2.0 ** -8 + 2.0 ** -20) * exact.abs() + 1e-30).all()
    if gate and not per_channel:
        z = ops.Partials(g.data[:, :, 4:4 + H * dv].contiguous())
        ops.delta_out(o, w, 1e-6, z, exact, H, dv)
        ops.delta_out(o, w, 1e-6, z, got, H, dv)
        assert (exact - got.float()).abs().le((2.0 ** -8 + 2.0 ** -20) * exact.abs() + 1e-30).all()
