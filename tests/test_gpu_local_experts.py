"""The fused path of an expert layer with all experts on one GPU, against the general formulation
(sort, grouped GEMMs, scatter-add) and a 64-bit oracle."""
import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu

from hyper_parallel_b200.ops import grouped, moe, native

# gate_up, activation and down products round to bf16 once each (2^-9 relative per element); the
# general path also rounds the gate and every partial sum of the combine
TOL = 2e-2


def _inputs(T, k, E, H, Fh, form):
    g = torch.Generator(device="cuda").manual_seed(T * 31 + E)

    def rn(*s, std=1.0):
        return (torch.randn(*s, device="cuda", generator=g) * std).to(torch.bfloat16)
    idx = torch.stack([torch.randperm(E, device="cuda", generator=g)[:k] for _ in range(T)])
    gate = torch.rand(T, k, device="cuda", generator=g) + 0.1
    x, w1, w2, dy = rn(T, H), rn(E, 2 * Fh, H, std=H ** -0.5), rn(E, H, Fh, std=Fh ** -0.5), rn(T, H)
    if form == "one_expert":
        idx = torch.full_like(idx, E - 1)                      # every pair, the slots of a token too
    elif form == "strided":
        idx = torch.stack([idx, idx], dim=-1)[..., 0]
        x = torch.cat([x, x], dim=1)[:, :H]
        dy = torch.cat([dy, dy], dim=1)[:, H:]
        gate = gate.t().contiguous().t()
    elif form == "offset":
        buf = torch.empty(T * H + 1, device="cuda", dtype=torch.bfloat16)
        buf[1:] = x.reshape(-1)
        x = buf[1:].view(T, H)                                  # contiguous, not 16-byte aligned
        gate = gate.to(torch.bfloat16)
    return x, idx, gate, w1, w2, dy


def _pass(fn, x, idx, gate, w1, w2, dy):
    leaves = [t.detach().requires_grad_() for t in (x, gate, w1, w2)]
    y = fn(leaves[0], idx, leaves[1], leaves[2], leaves[3], w1.shape[0])
    y.backward(dy)
    native.check_status()
    return [y.detach()] + [t.grad for t in leaves]


def _oracle(x, idx, gate, w1, w2, dy):
    leaves = [t.detach().double().requires_grad_() for t in (x, gate, w1, w2)]
    xd, gd, w1d, w2d = leaves
    y = torch.zeros_like(xd)
    for e in range(w1.shape[0]):
        tok, slot = (idx == e).nonzero(as_tuple=True)
        g, u = (xd[tok] @ w1d[e].t()).chunk(2, -1)
        y = y.index_add(0, tok, (F.silu(g) * u) @ w2d[e].t() * gd[tok, slot][:, None])
    y.backward(dy.double())
    return [y.detach()] + [t.grad if t.grad is not None else torch.zeros_like(t) for t in leaves]


def _err(a, b):
    return ((a.double() - b.double()).norm() / b.double().norm().clamp_min(1e-30)).item()


@pytest.mark.parametrize("form", ["plain", "one_expert", "strided", "offset"])
@pytest.mark.parametrize("T,k,E,H,Fh", [(1, 1, 1, 64, 8), (5, 2, 4, 136, 24), (77, 8, 32, 256, 128),
                                        (300, 4, 2, 512, 96), (127, 2, 1, 64, 64), (1000, 3, 8, 264, 136)])
def test_matches_general_path(monkeypatch, T, k, E, H, Fh, form):
    k = min(k, E)
    args = _inputs(T, k, E, H, Fh, form)
    assert grouped.local_experts_usable(args[0], args[1], args[2], args[3], args[4], E)
    got, again = _pass(moe.expert_parallel_ffn, *args), _pass(moe.expert_parallel_ffn, *args)
    monkeypatch.setattr(grouped, "local_experts_usable", lambda *a: False)
    general = _pass(moe.expert_parallel_ffn, *args)
    want = _oracle(*args)
    for a, b, c, d in zip(got, again, general, want):
        assert a.dtype == c.dtype and a.shape == c.shape
        assert torch.equal(a, b)                               # no atomics: the same bits on every run
        assert _err(a, d) < TOL and _err(a, d) <= 1.05 * _err(c, d) + 1e-6


@pytest.mark.parametrize("pad", [128, 256])
def test_both_layouts(monkeypatch, pad):
    monkeypatch.setattr(grouped, "_PAIR_MIN_ROWS", 0 if pad == 256 else 1 << 30)
    args = _inputs(391, 4, 6, 328, 72, "plain")
    for a, d in zip(_pass(moe.expert_parallel_ffn, *args), _oracle(*args)):
        assert _err(a, d) < TOL


@pytest.mark.parametrize("bad", [-1, 4])
def test_expert_id_out_of_range_is_refused(bad):
    args = list(_inputs(9, 2, 4, 64, 16, "plain"))
    args[1] = args[1].clone()
    args[1][3, 1] = bad
    with pytest.raises(ValueError, match="expert ids must lie in"):
        moe.expert_parallel_ffn(*args[:3], args[3], args[4], 4)
    good = _inputs(9, 2, 4, 64, 16, "plain")                   # nothing was launched on the bad ids
    assert _err(_pass(moe.expert_parallel_ffn, *good)[0], _oracle(*good)[0]) < TOL


def test_frozen_weights_and_inputs():
    x, idx, gate, w1, w2, dy = _inputs(33, 2, 4, 64, 16, "plain")
    want = _oracle(x, idx, gate, w1, w2, dy)
    for i, name in enumerate(("x", "gate", "w1", "w2")):
        leaves = [t.detach().requires_grad_(j == i) for j, t in enumerate((x, gate, w1, w2))]
        moe.expert_parallel_ffn(leaves[0], idx, leaves[1], leaves[2], leaves[3], 4).backward(dy)
        assert [t.grad is not None for t in leaves] == [j == i for j in range(4)], name
        assert _err(leaves[i].grad, want[i + 1]) < TOL


# ---- the gate weights are ordinary operands: higher derivatives, forward mode, batched gradients ----
def _toy(requires):
    x, idx, gate, w1, w2, dy = _inputs(23, 2, 4, 64, 16, "plain")
    return [t.requires_grad_(n in requires) for t, n in zip((x, gate, w1, w2), "xgab")], idx, dy


def _dense(x, idx, gate, w1, w2):
    """The layer in 64 bits."""
    xd, w1, w2 = x.double(), w1.double(), w2.double()
    y = 0
    for e in range(w1.shape[0]):
        g, u = (xd @ w1[e].t()).chunk(2, -1)
        y = y + (F.silu(g) * u) @ w2[e].t() * (gate.double() * (idx == e)).sum(-1, keepdim=True)
    return y


@pytest.mark.parametrize("requires", ["g", "xgab"])
def test_second_derivative_of_the_gate(requires):
    """A penalty on the gradient of the gate: its own derivatives, and those of the experts through one
    more (first-order) backward pass."""
    def penalty(fn, x, gate, w1, w2, idx):
        y = fn(x, idx, gate, w1, w2).double()
        (d,) = torch.autograd.grad((y * y).sum(), gate, create_graph=True)
        return (d.double() ** 2).sum()
    (x, gate, w1, w2), idx, _ = _toy(requires)
    penalty(lambda x, i, g, a, b: moe.expert_parallel_ffn(x, i, g, a, b, 4), x, gate, w1, w2, idx).backward()
    native.check_status()
    ref = [t.detach().double().requires_grad_(t.requires_grad) for t in (x, gate, w1, w2)]
    penalty(_dense, *ref, idx).backward()
    assert _err(gate.grad, ref[1].grad) < TOL
    if requires == "g":
        return
    # only the path through the gate's gradient has a graph (the experts' gradients do not): what the general
    # formulation gives for the inputs and weights is the same partial sum
    got = [t.grad.clone() for t in (x, w1, w2)]
    for t in (x, gate, w1, w2):
        t.grad = None
    general = pytest.MonkeyPatch()
    general.setattr(grouped, "local_experts_usable", lambda *a: False)
    try:
        penalty(lambda x, i, g, a, b: moe.expert_parallel_ffn(x, i, g, a, b, 4), x, gate, w1, w2, idx).backward()
    finally:
        general.undo()
    for a, t in zip(got, (x, w1, w2)):
        assert _err(a, t.grad) < 2 * TOL


def test_forward_mode_through_the_gate():
    (x, gate, w1, w2), idx, _ = _toy("")
    t = torch.randn_like(gate)
    with torch.autograd.forward_ad.dual_level():
        y = moe.expert_parallel_ffn(x, idx, torch.autograd.forward_ad.make_dual(gate, t), w1, w2, 4)
        primal, tangent = torch.autograd.forward_ad.unpack_dual(y)
    assert _err(primal, _dense(x, idx, gate, w1, w2)) < TOL
    assert _err(tangent, _dense(x, idx, t, w1, w2)) < TOL       # linear in the gate


def test_batched_gradients_of_the_gate():
    (x, gate, w1, w2), idx, dy = _toy("g")
    y = moe.expert_parallel_ffn(x, idx, gate, w1, w2, 4)
    dys = torch.stack([dy, -2 * dy])
    (got,) = torch.autograd.grad(y, gate, dys, is_grads_batched=True, retain_graph=True)
    (one,) = torch.autograd.grad(y, gate, dy)
    assert _err(got[0], one) < 1e-5 and _err(got[1], -2 * one) < 1e-5


def test_gate_overwritten_before_the_backward_pass():
    (x, gate, w1, w2), idx, dy = _toy("xab")
    want = _pass(moe.expert_parallel_ffn, x, idx, gate.clone(), w1, w2, dy)
    y = moe.expert_parallel_ffn(x, idx, gate, w1, w2, 4)
    gate.zero_()
    y.backward(dy)
    assert torch.equal(x.grad, want[1]) and torch.equal(w1.grad, want[3]) and torch.equal(w2.grad, want[4])


def test_calls_beyond_the_row_tables_take_the_general_path():
    """2^30 pairs and more do not fit the 32-bit tables (expanded inputs: nothing is allocated)."""
    x, idx, gate, w1, w2, _ = _inputs(1, 1, 2, 64, 16, "plain")
    assert grouped.local_experts_usable(x, idx, gate, w1, w2, 2)
    many = [t.expand(1 << 30, t.shape[1]) for t in (x, idx, gate)]
    assert not grouped.local_experts_usable(*many, w1, w2, 2)
