"""Strides of what the tensor functions allocate: those of torch.empty_like, also where a tensor counts as contiguous only
because a dimension has one element, and those of the operand where a kernel writes by them."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("view", [lambda x: x[:, :200], lambda x: x[:, :200].transpose(1, 2).contiguous().transpose(1, 2)])
def test_attention_output_has_the_strides_of_q(view):
    from byteir_b200 import ops
    gen = torch.Generator(device="cuda").manual_seed(1)
    base = [torch.randn((1, 256, 4, 64), generator=gen, device="cuda").to(torch.bfloat16) for _ in range(4)]
    q, k, v, x = (view(t) for t in base)
    out, lse = ops.flash_attn_fwd(q, k, v, 0.125, True)
    assert out.stride() == torch.empty_like(q).stride()
    do = torch.empty_like(q).copy_(x)
    grads = ops.flash_attn_bwd(do, q, k, v, out, lse, 0.125, True)
    plain = [t.contiguous().clone(memory_format=torch.contiguous_format) for t in (q, k, v, do)]
    out2, lse2 = ops.flash_attn_fwd(*plain[:3], 0.125, True)
    want = ops.flash_attn_bwd(plain[3].as_strided(out2.shape, out2.stride()), *plain[:3], out2, lse2, 0.125, True)
    for g, w in zip((out, lse) + grads, (out2, lse2) + want):
        assert torch.equal(g, w)


def test_scatter_add_output_has_the_strides_of_the_table():
    from byteir_b200 import ops
    x = torch.randn((1, 64, 32), device="cuda")[:, :50]
    out = ops.index_put_add(x, torch.arange(50, device="cuda"), torch.ones((50, 32), device="cuda"), dim=1)
    assert out.stride() == torch.empty_like(x).stride()
    assert torch.equal(out, x + 1)


# q, k and v as parts of one packed tensor: the gradients have their strides, and none is written past its end
def test_gradients_of_parts_of_a_packed_tensor():
    from byteir_b200 import ops
    gen = torch.Generator(device="cuda").manual_seed(2)
    packed = torch.randn((2, 300, 3, 4, 64), generator=gen, device="cuda").to(torch.bfloat16)
    do = torch.randn((2, 300, 4, 64), generator=gen, device="cuda").to(torch.bfloat16)
    q, k, v = packed.unbind(2)
    out, lse = ops.flash_attn_fwd(q, k, v, 0.125, True)
    grads = ops.flash_attn_bwd(do, q, k, v, out, lse, 0.125, True)
    plain = [t.contiguous() for t in (q, k, v)]
    out2, lse2 = ops.flash_attn_fwd(*plain, 0.125, True)
    for g, t, w in zip(grads, (q, k, v), ops.flash_attn_bwd(do, *plain, out2, lse2, 0.125, True)):
        assert g.stride() == t.stride() and torch.equal(g, w)
        assert g.untyped_storage().nbytes() >= 2 * (1 + sum((n - 1) * s for n, s in zip(t.shape, t.stride())))
    dpacked = torch.full_like(packed, 7.0)
    got = ops.flash_attn_bwd(do, q, k, v, out, lse, 0.125, True, dq=dpacked[:, :, 0], dk=dpacked[:, :, 1], dv=dpacked[:, :, 2])
    assert all(torch.equal(a, b) for a, b in zip(got, grads))
    with pytest.raises(ValueError):
        ops.flash_attn_bwd(do, q, k, v, out, lse, 0.125, True, dq=torch.empty_like(plain[0]))
