"""Backward of the fused residual add + RMS norm against float64."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# widths at the switches to two (2048) and four (8192) vectors per thread and the widest (16384), threads without a column, one
# vector; rows below and above the ring's depth and the grid
@pytest.mark.parametrize("rows,H", [(1, 8), (3, 264), (700, 264), (2401, 2048), (5, 2056), (1501, 3072), (447, 8192), (3, 8200),
                                    (701, 9216), (1, 16384), (301, 16384)])
@pytest.mark.parametrize("residual", [False, True])
def test_rms_norm_backward_matches_float64(rows, H, residual):
    from neuronx_distributed_llama3_2_b200.ops import norm

    g = torch.Generator(device="cuda").manual_seed(rows + H)

    def normal(*s):
        return torch.randn(*s, generator=g, device="cuda").bfloat16()

    x, r, w, dy, ds = (t.requires_grad_() for t in (normal(rows, H), normal(rows, H), normal(H), normal(rows, H), normal(rows, H)))
    if residual:
        torch.autograd.backward(norm.fused_add_rms_norm(x, r, w, 1e-6), (dy.detach(), ds.detach()))
        s = (x.detach() + r.detach()).double().requires_grad_()          # the stream is rounded once
    else:
        norm.rms_norm(x, w, 1e-6).backward(dy.detach())
        s = x.detach().double().requires_grad_()
    wd = w.detach().double().requires_grad_()
    y = s * torch.rsqrt(s.pow(2).mean(-1, keepdim=True) + 1e-6) * wd
    y.backward(dy.detach().double())
    want = s.grad + (ds.detach().double() if residual else 0.0)
    # dx: fp32 sums, one rounding to bf16 (at most 2^-8); the fp32 terms of dx cancel where it is small: 2^-18 of the largest
    assert ((x.grad.double() - want).abs() <= 2.0 ** -8 * want.abs() + 2.0 ** -18 * want.abs().max()).all()
    if residual:
        assert torch.equal(x.grad, r.grad)
    # dw: fp32 sums over the rows, then one rounding to bf16
    sums = (dy.detach().double() * s.detach() * torch.rsqrt(s.detach().pow(2).mean(-1, keepdim=True) + 1e-6)).abs().sum(0)
    assert ((w.grad.double() - wd.grad).abs() <= 2.0 ** -8 * wd.grad.abs() + 2.0 ** -20 * sums).all()


def test_rows_wider_than_the_ring_are_refused():
    from neuronx_distributed_llama3_2_b200.ops import norm

    x = torch.ones(2, 16392, device="cuda", dtype=torch.bfloat16).requires_grad_()
    with pytest.raises(RuntimeError, match="rmsnorm_bwd"):
        norm.rms_norm(x, x.detach()[0], 1e-6).sum().backward()
