"""Attention forward and backward at sequence lengths around the tiles of the kernels (2 or 16 tokens of the
row-statistics kernel: 16 above 18944 rows, 64 query rows, 128 key rows, 256 query rows per CTA), strided and packed inputs."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu

from hyper_parallel_b200.ops import attention, mla_attention, native

# bf16 probabilities and score gradients: 2^-9 per element, summed over rows; outputs round once more
TOL = 1e-2


def _err(a, b):
    return ((a.double() - b).norm() / b.norm().clamp_min(1e-30)).item()


def _oracle(q, k, v, do, causal, scale):
    q, k, v = (t.detach().double().requires_grad_() for t in (q, k, v))
    g = q.shape[2] // k.shape[2]
    s = torch.einsum("bihd,bjhd->bhij", q, k.repeat_interleave(g, 2)) * scale
    if causal:
        s = s.masked_fill(torch.ones(s.shape[-2:], dtype=torch.bool, device=s.device).triu(1), float("-inf"))
    o = torch.einsum("bhij,bjhd->bihd", torch.softmax(s, -1), v.repeat_interleave(g, 2))
    o.backward(do.double())
    return o.detach(), q.grad, k.grad, v.grad


@pytest.mark.parametrize("causal", [True, False])
@pytest.mark.parametrize("S,H,Hkv", [(1, 4, 2), (15, 4, 2), (17, 4, 2), (63, 4, 2), (65, 4, 2), (127, 4, 2), (129, 4, 2),
                                     (257, 4, 2), (400, 4, 2), (296, 32, 4), (301, 32, 4)])
def test_head_128(S, H, Hkv, causal):
    B = 2
    gen = torch.Generator(device="cuda").manual_seed(S)
    qkv = torch.randn(B, S, (H + 2 * Hkv) * 128, device="cuda", generator=gen).to(torch.bfloat16)
    q, k, v = (t.reshape(B, S, -1, 128) if S == 1 else t.view(B, S, -1, 128)
               for t in qkv.split([H * 128, Hkv * 128, Hkv * 128], dim=-1))
    do = torch.randn(B, S, H * 2, 128, device="cuda", generator=gen).to(torch.bfloat16)[:, :, :H]
    o, lse = attention.flash_attention_forward(q, k, v, causal=causal)
    dq, dk, dv = attention.flash_attention_backward(q, k, v, o, lse, do, causal=causal)
    native.check_status()
    want = _oracle(q, k, v, do, causal, 1 / math.sqrt(128))
    for got, ref in zip((o, dq, dk, dv), want):
        if S == 1 and ref.norm() < 1e-9:           # one key: no gradient through the softmax
            assert got.abs().max() < 1e-2
        else:
            assert _err(got, ref) < TOL


@pytest.mark.parametrize("S,H", [(1, 3), (15, 3), (17, 3), (65, 3), (129, 3), (300, 3), (301, 32)])
def test_latent(S, H):
    B = 2
    gen = torch.Generator(device="cuda").manual_seed(S)

    def rn(*shape):
        return torch.randn(*shape, device="cuda", generator=gen).to(torch.bfloat16)
    q, kv, kr, do = rn(B, S, H, 192), rn(B, S, H, 256), rn(B, S, 64), rn(B, S, H, 128)
    leaves = [t.detach().requires_grad_() for t in (q, kv, kr)]
    o = mla_attention.mla_attention(*leaves)
    o.backward(do)
    native.check_status()
    k = torch.cat([kv[..., :128], kr[:, :, None].expand(B, S, H, 64)], dim=-1)
    want = _oracle(q, k, kv[..., 128:], do, True, 1 / math.sqrt(192))
    assert _err(o, want[0]) < TOL
    dkv = torch.cat([want[2][..., :128], want[3]], dim=-1)
    assert _err(leaves[1].grad, dkv) < TOL
    if S > 1:
        assert _err(leaves[0].grad, want[1]) < TOL
        assert _err(leaves[2].grad, want[2][..., 128:].sum(2)) < TOL
