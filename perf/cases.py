"""Performance cases: the layers of a training step, each through the entry point a program calls.

A case is a dict of plain values.  ``prepare`` makes what a program holds before the call (weights,
activations, upstream gradients, an optimizer), ``run`` is one pass (forward and backward, or one
optimizer step) and returns every result of it, ``exact`` is the same computation in 64 bits in plain
torch.  Sizes are those of the configurations that the models, tests and benchmarks of this repository
name: Llama-3-8B (hidden 4096, 32 / 8 heads, ffn 14336, 128256 tokens), Llama-2-13B (5120, 40 / 40,
13824, 32000), DeepSeek-V3 (7168, 128 heads, low-rank 1536 / 512, ffn 18432, experts of 2048).
"""
from __future__ import annotations

import math

import torch
import torch.nn.functional as F
from torch.utils.checkpoint import checkpoint

from hyper_parallel_b200 import ops
from hyper_parallel_b200.models.deepseek_v3 import MLA, DeepSeekV3Config, DenseFFN
from hyper_parallel_b200.models.llama import Llama, LlamaBlock, LlamaConfig
from hyper_parallel_b200.ops import attention, moe
from hyper_parallel_b200.ops.flash_attention_score import flash_attention_score
from hyper_parallel_b200.optim import FusedAdamW

BF16 = torch.bfloat16
LLAMA = {"llama3_8b": LlamaConfig.llama3_8b, "llama2_13b": LlamaConfig.llama2_13b}


def listed():
    return [
        # the headline training step, layer by layer: 2 sequences of 4096 tokens
        {"name": "block_8b", "kind": "llama_block", "model": "llama3_8b", "batch": 2, "seq": 4096},
        # a short sequence alone on the GPU (fine-tuning on short prompts, small micro-batches)
        {"name": "block_8b_short", "kind": "llama_block", "model": "llama3_8b", "batch": 1, "seq": 203},
        # the output layer: final norm, vocabulary projection, loss and its gradients
        {"name": "lm_head_loss", "kind": "loss", "tokens": 8192, "hidden": 4096, "vocab": 128256},
        # the input layer: gather and dense weight gradient; token ids with the skew of text
        {"name": "embedding", "kind": "embedding", "tokens": 8192, "hidden": 4096, "vocab": 128256},
        # the optimizer on one block's worth of parameters
        {"name": "adamw", "kind": "adamw", "numel": 218112000, "tensors": 6},
        # grouped-query attention on a packed projection output, long sequence
        {"name": "attention_gqa", "kind": "attention", "batch": 1, "seq": 8192, "heads": 32, "kv_heads": 8},
        # the fused-attention operator of the reference's surface: full mask, BSH layout, odd length
        {"name": "attention_score", "kind": "attention_score", "batch": 3, "seq": 1531, "heads": 16,
         "kv_heads": 16, "layout": "BSH", "mode": 0},
        # the DeepSeek-V3 attention layer: low-rank projections, shared rotary key
        {"name": "mla_layer", "kind": "mla", "batch": 1, "seq": 4096, "fp8": False},
        # the dense feed-forward layer of DeepSeek-V3 with block-scaled fp8 forward products
        {"name": "ffn_fp8", "kind": "ffn", "tokens": 4096, "ffn": 18432, "fp8": True},
        # one expert-parallel rank's worth of routed experts, uneven load
        {"name": "moe_experts", "kind": "moe", "tokens": 4096, "experts": 32, "top_k": 8, "hidden": 7168,
         "ffn": 2048},
        # the same layer with few tokens: experts with a handful of rows or none
        {"name": "moe_experts_few", "kind": "moe", "tokens": 77, "experts": 32, "top_k": 8, "hidden": 7168,
         "ffn": 2048},
        # a whole small model, forward and backward: launches and host work count
        {"name": "tiny_model", "kind": "model", "batch": 2, "seq": 256, "layers": 2, "hidden": 512, "heads": 4,
         "kv_heads": 2, "ffn": 1024, "vocab": 1024},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["llama_block", "loss", "embedding", "adamw", "attention", "attention_score", "mla", "ffn",
                       "moe", "model"])
    if kind == "llama_block":
        batch = rng.choice([1, 2, 3])
        return {"kind": kind, "model": rng.choice(sorted(LLAMA)), "batch": batch,
                "seq": _log_int(rng, 64, 8192 // batch)}
    if kind == "loss":
        hidden, vocab = rng.choice([(4096, 128256), (5120, 32000), (7168, 129280), (4096, 50264)])
        return {"kind": kind, "tokens": _log_int(rng, 128, 4096 if hidden == 7168 else 8192), "hidden": hidden,
                "vocab": vocab}
    if kind == "embedding":
        hidden, vocab = rng.choice([(4096, 128256), (5120, 32000), (7168, 129280)])
        return {"kind": kind, "tokens": _log_int(rng, 64, 16384), "hidden": hidden, "vocab": vocab}
    if kind == "adamw":
        return {"kind": kind, "numel": _log_int(rng, 100000, 300000000), "tensors": rng.randint(1, 9)}
    if kind == "attention":
        batch = rng.choice([1, 2, 4])
        heads, kv = rng.choice([(32, 8), (40, 40), (16, 4), (8, 1)])
        return {"kind": kind, "batch": batch, "seq": _log_int(rng, 100, 8192 // batch), "heads": heads,
                "kv_heads": kv}
    if kind == "attention_score":
        batch = rng.choice([1, 2, 4])
        heads, kv = rng.choice([(32, 8), (16, 16), (8, 2)])
        return {"kind": kind, "batch": batch, "seq": _log_int(rng, 100, 8192 // batch), "heads": heads,
                "kv_heads": kv, "layout": rng.choice(["BSH", "SBH", "BNSD", "BSND"]), "mode": rng.choice([0, 2, 3])}
    if kind == "mla":
        batch = rng.choice([1, 2])
        return {"kind": kind, "batch": batch, "seq": _log_int(rng, 128, 4096 // batch),
                "fp8": rng.random() < 0.5}
    if kind == "ffn":
        return {"kind": kind, "tokens": _log_int(rng, 64, 4096), "ffn": rng.choice([18432, 2048]),
                "fp8": rng.random() < 0.7}
    if kind == "moe":
        hidden, ffn = rng.choice([(7168, 2048), (4096, 1408), (2048, 1024)])
        return {"kind": kind, "tokens": _log_int(rng, 16, 4096), "experts": rng.choice([8, 16, 32]),
                "top_k": rng.choice([2, 4, 8]), "hidden": hidden, "ffn": ffn}
    hidden = rng.choice([256, 512, 1024])
    return {"kind": "model", "batch": rng.choice([1, 2, 4]), "seq": rng.randint(33, 512), "layers": rng.randint(1, 4),
            "hidden": hidden, "heads": hidden // 128, "kv_heads": max(1, hidden // 256), "ffn": 2 * hidden,
            "vocab": rng.choice([512, 1024, 4096])}


# --------------------------------------------------------------- inputs --
class _Maker:
    """Random tensors of one seed."""

    def __init__(self, seed):
        self.gen = torch.Generator(device="cuda").manual_seed(seed)

    def randn(self, *shape, std=1.0, dtype=BF16):
        return torch.empty(shape, dtype=dtype, device="cuda").normal_(0.0, std, generator=self.gen)

    def uniform(self, *shape):
        return torch.empty(shape, dtype=torch.float32, device="cuda").uniform_(generator=self.gen)

    def norm_weight(self, *shape):
        return (1.0 + 0.1 * self.randn(*shape, dtype=torch.float32)).to(BF16)

    def zipf(self, n, vocab, offset=2.7):
        """Ids whose frequency falls like 1 / (rank + offset), as token frequencies of text do."""
        r = offset * torch.exp(self.uniform(n).double() * math.log((vocab + offset) / offset)) - offset
        return r.long().clamp_(0, vocab - 1)


def _fill(module, m, std):
    for p in module.parameters():
        with torch.no_grad():
            p.copy_(m.norm_weight(*p.shape) if p.dim() == 1 else m.randn(*p.shape, std=std))
    return module


def _llama_cfg(case):
    return LlamaConfig.tiny(vocab_size=case["vocab"], hidden_size=case["hidden"], num_layers=case["layers"],
                            num_heads=case["heads"], num_kv_heads=case["kv_heads"], head_dim=128,
                            ffn_size=case["ffn"])


def _score_shape(case, heads):
    b, s, n = case["batch"], case["seq"], heads
    return {"BSH": (b, s, n * 128), "SBH": (s, b, n * 128), "BNSD": (b, n, s, 128),
            "BSND": (b, s, n, 128)}[case["layout"]]


def prepare(case, seed):
    m = _Maker(seed)
    kind = case["kind"]
    if kind == "llama_block":
        cfg = LLAMA[case["model"]]()
        t = case["batch"] * case["seq"]
        return {"case": case, "cfg": cfg, "block": _fill(LlamaBlock(cfg, 0, device="cuda"), m, cfg.init_std),
                "h": m.randn(t, cfg.hidden_size), "resid": m.randn(t, cfg.hidden_size),
                "grads": [m.randn(t, cfg.hidden_size, std=0.01), m.randn(t, cfg.hidden_size, std=0.01)]}
    if kind == "loss":
        t, h, v = case["tokens"], case["hidden"], case["vocab"]
        target = m.zipf(t, v)
        target[m.uniform(t) < 0.02] = -100                    # prompt / padding positions carry no loss
        return {"case": case, "x": m.randn(t, h), "norm": m.norm_weight(h), "w": m.randn(v, h, std=0.02),
                "target": target}
    if kind == "embedding":
        t, h, v = case["tokens"], case["hidden"], case["vocab"]
        return {"case": case, "tokens": m.zipf(t, v), "w": m.randn(v, h, std=0.02), "grad": m.randn(t, h, std=0.01)}
    if kind == "adamw":
        params = []
        left, n = case["numel"], case["tensors"]
        for i in range(n):
            size = left if i == n - 1 else max(1, left // 2)
            left = max(1, left - size)
            p = torch.nn.Parameter(m.randn(size, std=0.02))
            p.grad = m.randn(size, std=1e-3)
            params.append(p)
        opt = FusedAdamW(params, lr=3e-4, betas=(0.9, 0.95), weight_decay=0.1)
        opt.init_state()
        for p in params:                                      # moments of a run under way
            st = opt.state[p]
            st["exp_avg"].copy_(m.randn(p.numel(), std=1e-3, dtype=torch.float32))
            st["exp_avg_sq"].copy_(m.randn(p.numel(), std=1e-3, dtype=torch.float32).square_())
        return {"case": case, "params": params, "opt": opt}
    if kind == "attention":
        w = (case["heads"] + 2 * case["kv_heads"]) * 128
        return {"case": case, "qkv": m.randn(case["batch"], case["seq"], w),
                "grad": m.randn(case["batch"], case["seq"], case["heads"], 128, std=0.01)}
    if kind == "attention_score":
        q, kv = _score_shape(case, case["heads"]), _score_shape(case, case["kv_heads"])
        return {"case": case, "q": m.randn(*q), "k": m.randn(*kv), "v": m.randn(*kv), "grad": m.randn(*q, std=0.01)}
    if kind == "mla":
        cfg = DeepSeekV3Config(fp8=case["fp8"])
        t = case["batch"] * case["seq"]
        return {"case": case, "cfg": cfg, "layer": _fill(MLA(cfg, device="cuda"), m, 0.02),
                "x": m.randn(t, cfg.hidden_size), "grad": m.randn(t, cfg.hidden_size, std=0.01)}
    if kind == "ffn":
        layer = DenseFFN(7168, case["ffn"], 0.02, device="cuda", fp8=case["fp8"])
        return {"case": case, "layer": _fill(layer, m, 0.02), "x": m.randn(case["tokens"], 7168),
                "grad": m.randn(case["tokens"], 7168, std=0.01)}
    if kind == "moe":
        t, e, k, h, f = (case[c] for c in ("tokens", "experts", "top_k", "hidden", "ffn"))
        # every token ranks the experts by its own scores plus the experts' popularity: uneven load
        score = m.randn(t, e, dtype=torch.float32) + 0.7 * m.randn(e, dtype=torch.float32)
        top = torch.sigmoid(score).topk(k, dim=-1)
        return {"case": case, "x": m.randn(t, h), "idx": top.indices,
                "gate": top.values / top.values.sum(-1, keepdim=True) * 2.5,
                "w_gate_up": m.randn(e, 2 * f, h, std=0.02), "w_down": m.randn(e, h, f, std=0.02),
                "grad": m.randn(t, h, std=0.01)}
    cfg = _llama_cfg(case)
    tokens = m.zipf(case["batch"] * (case["seq"] + 1), case["vocab"]).view(case["batch"], case["seq"] + 1)
    return {"case": case, "cfg": cfg, "model": _fill(Llama(cfg, device="cuda"), m, cfg.init_std),
            "inputs": tokens[:, :-1].contiguous(), "targets": tokens[:, 1:].contiguous()}


# ----------------------------------------------------------------- pass --
def _leaves(*tensors):
    """Fresh autograd leaves over the same memory, as the tensors of a new step are."""
    return [t.detach().requires_grad_() for t in tensors]


def _param_grads(module):
    return [p.grad for p in module.parameters()]


def _clear(module):
    for p in module.parameters():
        p.grad = None


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "llama_block":
        _clear(state["block"])
        h, resid = _leaves(state["h"], state["resid"])
        d, r = state["block"](h, resid, case["batch"], case["seq"])
        torch.autograd.backward([d, r], state["grads"])
        return [d.detach(), r.detach(), h.grad, resid.grad] + _param_grads(state["block"])
    if kind == "loss":
        x, norm, w = _leaves(state["x"], state["norm"], state["w"])
        logits = ops.linear(ops.rmsnorm(x, norm, 1e-5), w)
        loss = ops.fused_cross_entropy(logits, state["target"], unit_grad=True)
        loss.backward()
        return [loss.detach(), x.grad, norm.grad, w.grad]
    if kind == "embedding":
        (w,) = _leaves(state["w"])
        out = ops.embedding(state["tokens"], w)
        out.backward(state["grad"])
        return [out.detach(), w.grad]
    if kind == "adamw":
        state["opt"].step()
        out = []
        for p in state["params"]:
            st = state["opt"].state[p]
            out += [p.detach(), st["master"], st["exp_avg"], st["exp_avg_sq"]]
        return out
    if kind == "attention":
        (qkv,) = _leaves(state["qkv"])
        out = attention.causal_attention_packed(qkv, case["heads"], case["kv_heads"])
        out.backward(state["grad"])
        return [out.detach(), qkv.grad]
    if kind == "attention_score":
        q, k, v = _leaves(state["q"], state["k"], state["v"])
        out = flash_attention_score(q, k, v, case["heads"], case["layout"], scale=1.0 / math.sqrt(128),
                                    sparse_mode=case["mode"])[0]
        out.backward(state["grad"])
        return [out.detach(), q.grad, k.grad, v.grad]
    if kind == "mla":
        _clear(state["layer"])
        (x,) = _leaves(state["x"])
        out = state["layer"](x, case["batch"], case["seq"])
        out.backward(state["grad"])
        return [out.detach(), x.grad] + _param_grads(state["layer"])
    if kind == "ffn":
        _clear(state["layer"])
        (x,) = _leaves(state["x"])
        out = state["layer"](x)
        out.backward(state["grad"])
        return [out.detach(), x.grad] + _param_grads(state["layer"])
    if kind == "moe":
        x, gate, w1, w2 = _leaves(state["x"], state["gate"], state["w_gate_up"], state["w_down"])
        out = moe.expert_parallel_ffn(x, state["idx"], gate, w1, w2, case["experts"])
        out.backward(state["grad"])
        return [out.detach(), x.grad, gate.grad, w1.grad, w2.grad]
    _clear(state["model"])
    loss = state["model"](state["inputs"], state["targets"])
    loss.backward()
    return [loss.detach()] + _param_grads(state["model"])


# ----------------------------------------------------------------- work --
def _attention_flops(batch, seq, heads, dqk, dv, causal):
    """Products of the forward (QK, PV) and the backward (QK, dV, dP, dQ, dK) pass."""
    pairs = batch * heads * seq * (seq + 1) / 2 if causal else batch * heads * seq * seq
    return 2.0 * pairs * (4 * dqk + 3 * dv)


def work(case):
    kind = case["kind"]
    if kind == "llama_block":
        cfg = LLAMA[case["model"]]()
        h, t = cfg.hidden_size, case["batch"] * case["seq"]
        mats = h * (2 * cfg.num_heads + 2 * cfg.num_kv_heads) * cfg.head_dim + 3 * h * cfg.ffn_size
        flops = 6.0 * t * mats + _attention_flops(case["batch"], case["seq"], cfg.num_heads, 128, 128, True)
        return {"bytes": 2.0 * (2 * mats + 4 * h + 8 * t * h), "flops": flops}
    if kind == "loss":
        t, h, v = case["tokens"], case["hidden"], case["vocab"]
        return {"bytes": 2.0 * (2 * v * h + 2 * t * h + 2 * h) + 8 * t, "flops": 6.0 * t * h * v}
    if kind == "embedding":
        t, h, v = case["tokens"], case["hidden"], case["vocab"]
        rows = min(t, v)
        return {"bytes": 2.0 * (2 * rows * h + t * h + v * h) + 8 * t, "flops": 1.0 * t * h}
    if kind == "adamw":
        return {"bytes": 28.0 * case["numel"], "flops": 15.0 * case["numel"]}
    if kind in ("attention", "attention_score"):
        b, s, n, nkv = case["batch"], case["seq"], case["heads"], case["kv_heads"]
        causal = kind == "attention" or case["mode"] != 0
        return {"bytes": 2.0 * b * s * 128 * (2 * (n + 2 * nkv) + 2 * n),
                "flops": _attention_flops(b, s, n, 128, 128, causal)}
    if kind == "mla":
        c = DeepSeekV3Config()
        t, h, nh = case["batch"] * case["seq"], c.hidden_size, c.num_heads
        mats = h * (c.q_lora_rank + c.kv_lora_rank + 64) + nh * (192 * c.q_lora_rank + 256 * c.kv_lora_rank + 128 * h)
        return {"bytes": 2.0 * (2 * mats + 4 * t * h),
                "flops": 6.0 * t * mats + _attention_flops(case["batch"], case["seq"], nh, 192, 128, True)}
    if kind == "ffn":
        t, mats = case["tokens"], 3 * 7168 * case["ffn"]
        return {"bytes": 2.0 * (2 * mats + 4 * t * 7168), "flops": 6.0 * t * mats}
    if kind == "moe":
        t, e, k, h, f = (case[c] for c in ("tokens", "experts", "top_k", "hidden", "ffn"))
        return {"bytes": 2.0 * (2 * e * 3 * h * f + 4 * t * h) + 16.0 * t * k, "flops": 6.0 * t * k * 3 * h * f}
    cfg = _llama_cfg(case)
    t = case["batch"] * case["seq"]
    return {"bytes": 4.0 * cfg.num_params() + 16.0 * t, "flops": t * cfg.flops_per_token(case["seq"])}


def tolerance(case):
    kind = case["kind"]
    if kind == "embedding":
        return {"rel": 6e-3}          # one rounding to bf16 of an fp32 sum
    if kind == "adamw":
        return {"rel": 1e-4}          # fp32 update; a bf16 copy that may round the other way
    if kind in ("attention", "attention_score"):
        return {"rel": 1e-2}          # bf16 probabilities and score gradients
    if kind == "loss":
        return {"rel": 1e-2}          # bf16 logits and logit gradients
    if kind in ("mla", "ffn") and case["fp8"]:
        return {"rel": 7e-2}          # e4m3 operands that may round the other way
    if kind == "llama_block":
        return {"rel": 4e-2}          # as below, through attention and the residual stream
    return {"rel": 3e-2}              # bf16 activations through several products


# ---------------------------------------------------------------- exact --
def _d(t):
    return t.detach().double().requires_grad_()


def _grad(leaves):
    return [x.grad for x in leaves]


def _rmsnorm(x, w, eps):
    return x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + eps) * w


def _swiglu(gu):
    g, u = gu.chunk(2, dim=-1)
    return F.silu(g) * u


def _rope(x, seq, theta):
    """Rotate-half RoPE of ``x[T, N, D]``, position ``t % seq``."""
    t, _, d = x.shape
    pos = torch.arange(t, device=x.device, dtype=torch.float64) % seq
    inv = theta ** (-2.0 * torch.arange(d // 2, device=x.device, dtype=torch.float64) / d)
    ang = (pos[:, None] * inv)[:, None, :]
    a, b = x[..., :d // 2], x[..., d // 2:]
    return torch.cat([a * ang.cos() - b * ang.sin(), b * ang.cos() + a * ang.sin()], dim=-1)


def _one_head(q, k, v, scale, causal):
    s = q @ k.t() * scale
    if causal:
        s = s.masked_fill(torch.ones_like(s, dtype=torch.bool).triu(1), float("-inf"))
    return torch.softmax(s, dim=-1) @ v


def _attend(q, k, v, causal):
    """``q[B, S, H, D]``, ``k / v[B, S, Hkv, D]``; one head's scores at a time."""
    B, S, H, D = q.shape
    group = H // k.shape[2]
    heads = [[checkpoint(_one_head, q[b, :, h], k[b, :, h // group], v[b, :, h // group], 1.0 / math.sqrt(D), causal,
                         use_reentrant=False) for h in range(H)] for b in range(B)]
    return torch.stack([torch.stack(x, dim=1) for x in heads])


def _block(p, cfg, h, resid, batch, seq):
    attn_norm, wqkv, wo, ffn_norm, w_gate_up, w_down = p
    nh, nkv, hd = cfg.num_heads, cfg.num_kv_heads, cfg.head_dim
    t = batch * seq
    if resid is not None:
        h = h + resid
    qkv = _rmsnorm(h, attn_norm, cfg.norm_eps) @ wqkv.t()
    q, k, v = qkv.split([nh * hd, nkv * hd, nkv * hd], dim=-1)
    q = _rope(q.reshape(t, nh, hd), seq, cfg.rope_theta).view(batch, seq, nh, hd)
    k = _rope(k.reshape(t, nkv, hd), seq, cfg.rope_theta).view(batch, seq, nkv, hd)
    a = _attend(q, k, v.reshape(batch, seq, nkv, hd), True)
    h = h + a.reshape(t, nh * hd) @ wo.t()
    return _swiglu(_rmsnorm(h, ffn_norm, cfg.norm_eps) @ w_gate_up.t()) @ w_down.t(), h


class _Quantised(torch.autograd.Function):
    """``x @ w.T`` on operands rounded to e4m3 with one scale per 1x128 (x) and 128x128 (w) tile;
    the gradients are those of the unrounded product (the layer's definition)."""

    @staticmethod
    def forward(ctx, x, w):
        ctx.save_for_backward(x, w)
        m, k = x.shape
        n = w.shape[0]
        xb = x.view(m, k // 128, 128)
        sx = xb.abs().amax(-1, keepdim=True).clamp_min(1e-10) / 448.0
        xq = ((xb / sx).float().to(torch.float8_e4m3fn).double() * sx).view(m, k)
        wb = F.pad(w, (0, 0, 0, -n % 128)).view(-1, 128, k // 128, 128)
        sw = wb.abs().amax(dim=(1, 3), keepdim=True).clamp_min(1e-10) / 448.0
        wq = ((wb / sw).float().to(torch.float8_e4m3fn).double() * sw).view(-1, k)[:n]
        return xq @ wq.t()

    @staticmethod
    def backward(ctx, dy):
        x, w = ctx.saved_tensors
        return dy @ w, dy.t() @ x


def _lin(x, w, fp8):
    return _Quantised.apply(x.contiguous(), w) if fp8 else x @ w.t()


def _mla(layer, c, x, batch, seq, fp8):
    wq_a, q_norm, wq_b, wkv_a, kv_norm, wkv_b, wo = layer
    t, nh, dn, dr, dv = x.shape[0], c.num_heads, c.qk_nope_head_dim, c.qk_rope_head_dim, c.v_head_dim
    q = _lin(_rmsnorm(_lin(x, wq_a, fp8), q_norm, c.norm_eps), wq_b, fp8).view(t, nh, dn + dr)
    q = torch.cat([q[..., :dn], _rope(q[..., dn:], seq, c.rope_theta)], dim=-1)
    kv_c, k_rope = _lin(x, wkv_a, fp8).split([c.kv_lora_rank, dr], dim=-1)
    k_rope = _rope(k_rope.reshape(t, 1, dr), seq, c.rope_theta)
    kv = _lin(_rmsnorm(kv_c, kv_norm, c.norm_eps), wkv_b, fp8).view(t, nh, dn + dv)
    k = torch.cat([kv[..., :dn], k_rope.expand(t, nh, dr)], dim=-1)
    o = _attend(q.view(batch, seq, nh, dn + dr), k.view(batch, seq, nh, dn + dr),
                kv[..., dn:].reshape(batch, seq, nh, dv), True)
    return _lin(o.reshape(t, nh * dv), wo, fp8)


def exact(case, seed):
    state = prepare(case, seed)
    kind = case["kind"]
    if kind == "llama_block":
        p = [_d(x) for x in state["block"].parameters()]
        h, resid = _d(state["h"]), _d(state["resid"])
        d, r = _block(p, state["cfg"], h, resid, case["batch"], case["seq"])
        torch.autograd.backward([d, r], [g.double() for g in state["grads"]])
        return [d.detach(), r.detach(), h.grad, resid.grad] + _grad(p)
    if kind == "loss":
        x, norm, w = _d(state["x"]), _d(state["norm"]), _d(state["w"])
        logits = _rmsnorm(x, norm, 1e-5) @ w.t()
        loss = F.cross_entropy(logits, state["target"], ignore_index=-100, reduction="sum") / case["tokens"]
        loss.backward()
        return [loss.detach()] + _grad([x, norm, w])
    if kind == "embedding":
        w = state["w"]
        dw = torch.zeros(w.shape, dtype=torch.float64, device=w.device)
        dw.index_add_(0, state["tokens"], state["grad"].double())
        return [w[state["tokens"]].double(), dw]
    if kind == "adamw":
        out = []
        for p in state["params"]:
            st = state["opt"].state[p]
            g = p.grad.double()
            m = 0.9 * st["exp_avg"].double() + (1 - 0.9) * g
            v = 0.95 * st["exp_avg_sq"].double() + (1 - 0.95) * g * g
            upd = (m / (1 - 0.9)) / ((v / (1 - 0.95)).sqrt() + 1e-8)
            w = st["master"].double() * (1 - 3e-4 * 0.1) - 3e-4 * upd
            out += [None, w, m, v]                            # the bf16 copy is the master, rounded
        return out
    if kind == "attention":
        qkv = _d(state["qkv"])
        b, s, n, nkv = case["batch"], case["seq"], case["heads"], case["kv_heads"]
        q, k, v = qkv.view(b, s, n + 2 * nkv, 128).split([n, nkv, nkv], dim=2)
        out = _attend(q, k, v, True)
        out.backward(state["grad"].double())
        return [out.detach(), qkv.grad]
    if kind == "attention_score":
        q, k, v = _d(state["q"]), _d(state["k"]), _d(state["v"])
        layout, b, s = case["layout"], case["batch"], case["seq"]

        def split(t, n):
            if layout == "BNSD":
                return t.transpose(1, 2)
            return (t.transpose(0, 1) if layout == "SBH" else t).reshape(b, s, n, 128)
        out = _attend(split(q, case["heads"]), split(k, case["kv_heads"]), split(v, case["kv_heads"]),
                      case["mode"] != 0)
        if layout == "BNSD":
            out = out.transpose(1, 2)
        elif layout == "SBH":
            out = out.reshape(b, s, -1).transpose(0, 1)
        elif layout == "BSH":
            out = out.reshape(b, s, -1)
        out.backward(state["grad"].double())
        return [out.detach()] + _grad([q, k, v])
    if kind == "mla":
        p, x = [_d(w) for w in state["layer"].parameters()], _d(state["x"])
        out = _mla(p, state["cfg"], x, case["batch"], case["seq"], case["fp8"])
        out.backward(state["grad"].double())
        return [out.detach()] + _grad([x] + p)
    if kind == "ffn":
        p, x = [_d(w) for w in state["layer"].parameters()], _d(state["x"])
        out = _lin(_swiglu(_lin(x, p[0], case["fp8"])), p[1], case["fp8"])
        out.backward(state["grad"].double())
        return [out.detach()] + _grad([x] + p)
    if kind == "moe":
        x, gate = state["x"].double(), state["gate"].double()
        grad, idx = state["grad"].double(), state["idx"]
        out, dx, dgate = torch.zeros_like(x), torch.zeros_like(x), torch.zeros_like(gate)
        dw1, dw2 = [], []
        for e in range(case["experts"]):                      # one expert's 64-bit weights at a time
            tok, slot = (idx == e).nonzero(as_tuple=True)
            w1, w2 = _d(state["w_gate_up"][e]), _d(state["w_down"][e])
            xe, ge = _d(x[tok]), _d(gate[tok, slot])
            ye = _swiglu(xe @ w1.t()) @ w2.t() * ge[:, None]
            ye.backward(grad[tok])
            out.index_add_(0, tok, ye.detach())
            dx.index_add_(0, tok, xe.grad)
            dgate[tok, slot] = ge.grad
            dw1.append(w1.grad)
            dw2.append(w2.grad)
        return [out, dx, dgate, torch.stack(dw1), torch.stack(dw2)]
    cfg, model = state["cfg"], state["model"]
    p = {n: _d(w) for n, w in model.named_parameters()}
    h, resid = p["embed"][state["inputs"].reshape(-1)], None
    for i in range(cfg.num_layers):
        names = ("attn_norm", "wqkv", "wo", "ffn_norm", "w_gate_up", "w_down")
        h, resid = _block([p[f"layers.{i}.{n}"] for n in names], cfg, h, resid, case["batch"], case["seq"])
    logits = _rmsnorm(h + resid, p["final_norm"], cfg.norm_eps) @ p["lm_head"].t()
    loss = F.cross_entropy(logits, state["targets"].reshape(-1))
    loss.backward()
    return [loss.detach()] + [w.grad for w in p.values()]
