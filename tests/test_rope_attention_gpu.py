"""Rotation in and out of place, and rotation + attention as one autograd node, against fp32."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _tables(n, D):
    from neuronx_distributed_llama3_2_b200.ops.rope import build_rope_cache

    return build_rope_cache(n, D, 10000.0, None, device="cuda")


# heads around the four that a thread takes, with copied heads behind them; the smallest head size and one that is no power of two
@pytest.mark.parametrize("T,heads,rot,D", [(1, 1, 1, 16), (7, 5, 3, 48), (33, 9, 8, 64), (130, 6, 0, 128), (1001, 40, 32, 128),
                                             (1700, 19, 17, 128)])
@pytest.mark.parametrize("offset", [0, 1])
def test_rope_matches_fp32(T, heads, rot, D, offset):
    from neuronx_distributed_llama3_2_b200.ops import rope

    g = torch.Generator(device="cuda").manual_seed(T)
    x = torch.randn(T * heads * D + offset, generator=g, device="cuda").bfloat16()[offset:].view(T, heads, D)
    cos, sin = _tables(T, D)
    ref = rope.rope_ref(x.float(), cos, sin, rot, 2, T)
    xg = x.detach().requires_grad_()
    y = rope.apply_rope(xg, cos, sin, rot, 2, T)
    y.backward(y.detach())
    back = rope.rope_ref(y.detach().float(), cos, sin, rot, 2, T, inverse=True)
    # one rounding to bf16: at most 2^-8 of the value (and of the two products, in fp32, 2^-22)
    for got, want in ((y, ref), (xg.grad, back), (rope.rope_inplace_(x.clone(), cos, sin, rot, 2, T), ref)):
        assert ((got.float() - want).abs() <= 2.0 ** -8 * want.abs() + 2.0 ** -20).all()
    assert torch.equal(y[:, rot:], x[:, rot:])


@pytest.mark.parametrize("S,B,n_q,n_kv,D", [(1, 1, 2, 1, 64), (65, 3, 6, 2, 64), (257, 2, 3, 3, 128), (700, 1, 8, 2, 128)])
def test_rope_attention_matches_fp32(S, B, n_q, n_kv, D):
    from neuronx_distributed_llama3_2_b200.ops import attention, rope

    g = torch.Generator(device="cuda").manual_seed(S)
    heads = n_q + 2 * n_kv
    x = torch.randn(S, B, heads, D, generator=g, device="cuda").bfloat16()
    d = torch.randn(B, n_q, S, D, generator=g, device="cuda").bfloat16()
    cos, sin = _tables(S, D)
    xg = x.detach().requires_grad_()
    o = attention.rope_flash_attn_func(xg, cos, sin, n_q, n_kv)
    o.backward(d)
    assert o.permute(2, 0, 1, 3).is_contiguous()
    xr = x.double().requires_grad_()
    r = rope.rope_ref(xr.view(S * B, heads, D), cos, sin, n_q + n_kv, B, S).view(S, B, heads, D).permute(1, 2, 0, 3)
    ref = attention.attention_ref(r[:, :n_q], r[:, n_q:n_q + n_kv], r[:, n_q + n_kv:], True)
    ref.backward(d.to(ref.dtype))
    # roundings to bf16, at most 2^-8 of a value each: forward the rotated heads, the probabilities and the output; backward also
    # the score gradients, dq / dk / dv, and their rotation back
    assert (o.double() - ref).norm() <= 3 * 2.0 ** -8 * ref.norm()
    assert (xg.grad.double() - xr.grad).norm() <= 6 * 2.0 ** -8 * xr.grad.norm()
