"""Cross entropy kernels (row in registers, row streamed twice): remainders and special values."""
import pytest
import torch

pytestmark = pytest.mark.gpu

from hyper_parallel_b200.ops import functional as Fn
from hyper_parallel_b200.ops import native


def _pad8(v):
    return (v + 7) // 8 * 8


# 128 threads x 1 / 2 / 4 / 8 vectors in registers, streamed rows from 8193 logits on
@pytest.mark.parametrize("V", [1, 7, 8, 1023, 1024, 1032, 2049, 4100, 8192, 8200, 32768, 32775, 32776, 36865,
                               50257, 128256, 270001])
def test_against_64_bits(V):
    gen = torch.Generator(device="cuda").manual_seed(V)
    T, ld = 13, _pad8(V) + 8
    buf = (torch.randn(T, ld, device="cuda", generator=gen) * 3).to(torch.bfloat16)
    tgt = torch.randint(0, V, (T,), device="cuda", generator=gen)
    tgt[0], tgt[1], tgt[2], tgt[3], tgt[4] = 0, V - 1, -100, V, min(V - 1, V // 8 * 8)
    before = buf.clone()
    logits = buf[:, :V]
    x = logits.double().requires_grad_()
    ignored = (tgt < 0) | (tgt >= V)
    want = torch.nn.functional.cross_entropy(x, tgt.masked_fill(ignored, -100), ignore_index=-100, reduction="none")
    (want.sum() * 0.25).backward()
    loss = Fn.cross_entropy_fwd_bwd(logits, tgt, 0.25)
    native.check_status()
    # fp32 log-sum-exp: a few units of 2^-24 times its size; gradients round to bf16 once
    assert (loss.double() - want.detach()).abs().max() < 1e-5 * (1 + want.detach().abs().max())
    err = (logits.double() - x.grad).norm() / x.grad.norm().clamp_min(1e-30)
    assert err < 2.0 ** -8 if V > 1 else logits.abs().max() < 1e-6
    assert (logits[ignored] == 0).all()
    assert torch.equal(buf[:, V:], before[:, V:])


@pytest.mark.parametrize("V", [1000, 40000, 128256])
def test_masked_and_non_finite_logits(V):
    base = torch.randn(6, V, device="cuda").to(torch.bfloat16)
    base[0, : V // 2] = float("-inf")                        # masked by -inf, whole vectors of a thread
    base[1, :] = -3e38
    base[2] = float("-inf")
    base[3, V // 3] = float("inf")
    base[4, V - 1] = float("nan")
    base[5, 1:] = float("-inf")
    tgt = torch.tensor([V - 1, 5, 5, 5, 5, 0], device="cuda")
    x = base.double()
    want = torch.logsumexp(x, -1) - x.gather(1, tgt[:, None])[:, 0]
    got = base.clone()
    loss = Fn.cross_entropy_fwd_bwd(got, tgt, 1.0)
    native.check_status()
    # row 1: the log-sum-exp of a row at -3e38 is that value in fp32 (log V is lost), as it always was
    assert torch.isfinite(loss[1]) and torch.isfinite(got[1].float()).all()
    for row in (0, 5):
        assert abs(loss[row].item() - want[row].item()) < 1e-4 * (1 + abs(want[row].item()))
        g = torch.softmax(x[row], -1)
        g[tgt[row]] -= 1
        assert (got[row].double() - g).abs().max() < 2.0 ** -8
    for row in (2, 3, 4):                                    # no finite answer: NaN throughout
        assert torch.isnan(loss[row]) and torch.isnan(got[row].float()).any()


@pytest.mark.parametrize("V,T,sms", [(8200, 13, 1), (16392, 13, 1), (32775, 13, 1), (128256, 7, 1), (8200, 0, 0),
                                     (16392, 0, 0), (32775, 0, 0)])
def test_several_rows_per_cta(V, T, sms):
    """The streaming kernel's walk: the producer runs ahead into the next row, whose stages and phases go on
    where the row before left them (2 copies per 16384 logits over 3 stages).  ``sms`` = 1 puts all rows on two
    CTAs; 0: the whole GPU with five rows for most CTAs."""
    sms = sms or native.sm_count("cuda")
    T = T or 5 * 2 * sms + 3
    gen = torch.Generator(device="cuda").manual_seed(V + T)
    ld = _pad8(V)
    buf = (torch.randn(T, ld, device="cuda", generator=gen) * 3).to(torch.bfloat16)
    buf[5::7, : V // 3] = float("-inf")
    dead = torch.zeros(T, dtype=torch.bool, device="cuda")
    dead[3::11] = True
    buf[dead] = float("-inf")                                # no finite logit: NaN, and nothing of it in the rows around
    tgt = torch.randint(V // 3, V, (T,), device="cuda", generator=gen)
    tgt[2::5] = -100
    before, logits = buf.clone(), buf[:, :V]
    loss = torch.empty(T, device="cuda")
    native.check(native.lib().hpb_cross_entropy(logits.data_ptr(), tgt.data_ptr(), loss.data_ptr(), T, V, ld, 0.5,
                                                native.status_word("cuda").data_ptr(), sms, native.stream()), "ce")
    native.check_status()
    ignored = tgt < 0
    worst = 0.0
    for t0 in range(0, T, 64):                               # (64 bits: a few rows at a time)
        rows = slice(t0, min(t0 + 64, T))
        x = before[rows, :V].double()
        want = torch.logsumexp(x, -1) - x.gather(1, tgt[rows].clamp_min(0)[:, None])[:, 0]
        grad = torch.softmax(x, -1)
        grad.scatter_add_(1, tgt[rows].clamp_min(0)[:, None], torch.full((x.shape[0], 1), -1.0, device="cuda", dtype=x.dtype))
        live = ~ignored[rows] & ~dead[rows]
        assert (loss[rows].double() - want)[live].abs().max() < 1e-5 * (1 + want[live].abs().max())
        got = logits[rows].double()
        err = (got - 0.5 * grad)[live].norm(dim=-1) / (0.5 * grad)[live].norm(dim=-1)
        worst = max(worst, err.max().item())
        quiet = ignored[rows] & ~dead[rows]
        assert (got[quiet] == 0).all() and (loss[rows][quiet] == 0).all()
        assert torch.isnan(loss[rows][dead[rows] & ~ignored[rows]]).all()
    assert worst < 2.0 ** -8                                 # one rounding to bf16
    assert torch.equal(buf[:, V:], before[:, V:])
