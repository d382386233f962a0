"""The packed in-place rotary tail equals the one on the per-head view, values and gradients."""
import pytest
import torch

from hyper_parallel_b200.ops import mla_attention


@pytest.mark.parametrize("T,NH,D,dr,S", [(1, 1, 32, 16, 1), (12, 3, 48, 16, 4), (10, 2, 192, 64, 5)])
def test_packed_equals_view(T, NH, D, dr, S):
    torch.manual_seed(T)
    x, dy = torch.randn(T, NH * D), torch.randn(T, NH * D)
    a, b = x.clone().requires_grad_(), x.clone().requires_grad_()
    ya = mla_attention.rope_tail_((a * 1.0).view(T, NH, D), dr, S, 10000.0).reshape(T, NH * D)
    yb = mla_attention.rope_tail_packed_(b * 1.0, NH, dr, S, 10000.0)
    assert torch.equal(ya, yb)
    ya.backward(dy)
    yb.backward(dy)
    assert torch.equal(a.grad, b.grad)


def test_no_tokens():
    x = torch.zeros(0, 3 * 48, requires_grad=True)
    y = mla_attention.rope_tail_packed_(x * 1.0, 3, 16, 4, 10000.0)
    y.backward(torch.zeros_like(y))
    assert y.shape == (0, 144) and x.grad.shape == (0, 144)
