"""The work a user of this framework has it do, as timed cases.

Six kinds, each through the entry points that the model classes and library callers use:

  step     one decode step of a quantised decoder (DecodeSession: the replayed CUDA graph), sequences of ragged lengths
  mlp      rms norm + fused gate|up (silu * mul) + down projection into the fp32 residual stream, 4- or 8-bit weights
  decode   rope + cache append + attention of one new token per sequence over a filled cache
  prompt   the same for a portion of a prompt (causal, behind what the cache already holds)
  experts  routed experts with a shared expert (dense 16-bit weights), from decode batches to prompts
  delta    a gated-delta-rule mixer with per-channel decays over a ragged batch of prompts

Widths, head counts and bit widths are those of this repository's configurations (synth.CONFIGS and the design sizes of
bench.py); batch sizes, context lengths and prompt lengths range from one sequence to a full server batch.
"""
import math

import torch

from mlx_parallm_b200 import ops
from mlx_parallm_b200._lib import EPI_ADD_RESIDUAL, EPI_SILU_MUL
from mlx_parallm_b200.models import llama, qwen3
from mlx_parallm_b200.models._sequence import GatedDeltaMixer, GatedFF, RoutedExperts, Scratch
from mlx_parallm_b200.models._transformer import QuantizedLinear, advance_cache, prepare_cache
from mlx_parallm_b200.models.base import DeltaRuleState
from mlx_parallm_b200.synth import get_config
from mlx_parallm_b200.utils import DecodeSession

DEV = "cuda"
DT = {"f16": torch.float16, "bf16": torch.bfloat16}
GROUP = 64
EPS = 1e-5
ARCHS = ("mistral-7b", "llama-3-8b", "qwen3-14b")
DELTA_EPS = 1e-6
TAPS = 4


def listed():
    return [
        # one user's chat: latency of a single sequence's decode step
        dict(name="step-b1", kind="step", arch="mistral-7b", layers=4, dtype="f16", batch=1, context=1000),
        # a full server batch of short conversations: weights, many small kernels, a large head
        dict(name="step-b64", kind="step", arch="qwen3-14b", layers=4, dtype="bf16", batch=64, context=500),
        # the weights-bound block of a single sequence
        dict(name="mlp-1", kind="mlp", hidden=4096, inter=14336, bits=4, dtype="f16", rows=1),
        # ... of a moderate decode batch
        dict(name="mlp-24", kind="mlp", hidden=5120, inter=17408, bits=4, dtype="bf16", rows=24),
        # ... of a short prompt or a large batch, rows that fill no tile
        dict(name="mlp-8bit-201", kind="mlp", hidden=8192, inter=28672, bits=8, dtype="bf16", rows=201),
        # ... of a chunk of a long prompt
        dict(name="mlp-4096", kind="mlp", hidden=4096, inter=14336, bits=4, dtype="f16", rows=4096),
        # attention of a decode batch over long contexts: the cache stream
        dict(name="decode-16x8k", kind="decode", heads=32, kv_heads=8, qk_norm=False, dtype="f16", batch=16, context=8192),
        # prompts of a small batch, odd length, empty cache
        dict(name="prompt-4x777", kind="prompt", heads=32, kv_heads=8, qk_norm=False, dtype="f16", batch=4, tokens=777, context=0),
        # a portion of a long prompt behind what is already cached
        dict(name="prompt-4k-at-4k", kind="prompt", heads=40, kv_heads=8, qk_norm=True, dtype="bf16", batch=1, tokens=4096, context=4096),
        # routed experts of a decode batch and of prompts
        dict(name="experts-32", kind="experts", width=2048, ff=2048, experts=16, top=2, shared=4096, dtype="bf16", tokens=32),
        dict(name="experts-6000", kind="experts", width=2048, ff=2048, experts=16, top=2, shared=4096, dtype="bf16", tokens=6000),
        # a recurrent layer over a batch of prompts
        dict(name="delta-4x512", kind="delta", width=2048, heads=16, kv_heads=8, dim=128, dtype="bf16", batch=4, tokens=512),
    ]


def _log(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["step", "mlp", "mlp", "mlp", "decode", "prompt", "prompt", "experts", "delta"])
    dtype = rng.choice(["f16", "bf16"])
    if kind == "step":
        return dict(kind=kind, arch=rng.choice(ARCHS), layers=rng.randint(2, 4), dtype=dtype, batch=_log(rng, 1, 64),
                    context=_log(rng, 16, 1000))
    if kind == "mlp":
        hidden, inter, bits = rng.choice([(4096, 14336, 4), (5120, 17408, 4), (4096, 14336, 8), (8192, 28672, 8)])
        return dict(kind=kind, hidden=hidden, inter=inter, bits=bits, dtype=dtype, rows=_log(rng, 1, 1024 if hidden == 8192 else 3000))
    if kind in ("decode", "prompt"):
        heads, kv_heads, norm = rng.choice([(32, 8, False), (40, 8, True), (64, 8, False)])
        case = dict(kind=kind, heads=heads, kv_heads=kv_heads, qk_norm=norm, dtype=dtype)
        if kind == "decode":
            batch = _log(rng, 1, 64)
            return dict(case, batch=batch, context=_log(rng, 64, min(16384, 131072 // batch)))
        batch = _log(rng, 1, 8)
        tokens = _log(rng, 2, min(4096, 8192 // batch))
        return dict(case, batch=batch, tokens=tokens, context=rng.choice([0, _log(rng, 16, 2048)]))
    if kind == "experts":
        width, ff = rng.choice([(2048, 2048), (4096, 3584)])
        return dict(kind=kind, width=width, ff=ff, experts=rng.choice([8, 16, 32]), top=rng.choice([1, 2, 4]), shared=rng.choice([0, 2 * ff]),
                    dtype="bf16", tokens=_log(rng, 1, 6000 if width == 2048 else 1500))
    width, heads = rng.choice([(2048, 16), (4096, 32)])
    batch = _log(rng, 1, 16)
    return dict(kind=kind, width=width, heads=heads, kv_heads=8, dim=128, dtype="bf16", batch=batch, tokens=_log(rng, 1, min(600, 4096 // batch)))


# ---------------------------------------------------------------------------------------------------------------------
# inputs, in plain torch, from the seed alone
class _Source:
    def __init__(self, seed):
        self.g = torch.Generator(device=DEV)
        self.g.manual_seed(int(seed) * 7919 + 13)

    def normal(self, *shape):
        return torch.randn(shape, generator=self.g, device=DEV)

    def uniform(self, *shape):
        return torch.rand(shape, generator=self.g, device=DEV)

    def ints(self, hi, *shape):
        return torch.randint(0, hi, shape, generator=self.g, device=DEV)

    def quantised(self, n, k, bits, dt, gain=1.0):
        """Packed codes, signed group scales and biases of an n x k matrix with entries of about 1 / sqrt(k)."""
        top = float((1 << bits) - 1)
        w = torch.randint(-(2 ** 31), 2 ** 31, (n, k * bits // 32), generator=self.g, device=DEV, dtype=torch.int64).to(torch.int32)
        mag = (self.uniform(n, k // GROUP) + 0.5) * (2.0 * gain / top) / math.sqrt(k)
        s = torch.where(self.uniform(n, k // GROUP) < 0.5, -mag, mag).to(dt)
        b = (-s.float() * (top / 2) + self.normal(n, k // GROUP) * (0.01 * gain / math.sqrt(k))).to(dt)
        return w, s, b

    def matrix(self, n, k, dt):
        return (self.normal(n, k) / math.sqrt(k)).to(dt)

    def norm(self, n, dt):
        return (1.0 + 0.02 * self.normal(n)).to(dt)

    def lengths(self, batch, most):
        """Ragged: between half of ``most`` and ``most`` (0 stays 0)."""
        return (most // 2 + (self.uniform(batch) * (most - most // 2 + 1)).long().clamp(max=most - most // 2)).to(torch.int32)


def _step_cfg(case):
    return get_config(case["arch"], num_hidden_layers=case["layers"])


def _step_inputs(case, seed):
    src, cfg, dt = _Source(seed), _step_cfg(case), DT[case["dtype"]]
    h, inter, V = cfg["hidden_size"], cfg["intermediate_size"], cfg["vocab_size"]
    D = cfg.get("head_dim") or h // cfg["num_attention_heads"]
    Hq, Hkv, bits = cfg["num_attention_heads"], cfg["num_key_value_heads"], cfg["quantization"]["bits"]
    w = {}

    def put(name, n, k, gain=1.0):
        for leaf, t in zip(("weight", "scales", "biases"), src.quantised(n, k, bits, dt, gain)):
            w[name + "." + leaf] = t

    put("model.embed_tokens", V, h, 0.5 * math.sqrt(h))
    put("lm_head", V, h)
    w["model.norm.weight"] = src.norm(h, dt)
    for i in range(cfg["num_hidden_layers"]):
        p = f"model.layers.{i}."
        for nm, n, k in (("self_attn.q_proj", Hq * D, h), ("self_attn.k_proj", Hkv * D, h), ("self_attn.v_proj", Hkv * D, h),
                         ("self_attn.o_proj", h, Hq * D), ("mlp.gate_proj", inter, h), ("mlp.up_proj", inter, h), ("mlp.down_proj", h, inter)):
            put(p + nm, n, k)
        w[p + "input_layernorm.weight"], w[p + "post_attention_layernorm.weight"] = src.norm(h, dt), src.norm(h, dt)
        if cfg["model_type"] == "qwen3":
            w[p + "self_attn.q_norm.weight"], w[p + "self_attn.k_norm.weight"] = src.norm(D, dt), src.norm(D, dt)
    B, T = case["batch"], case["context"]
    kv = [(src.normal(B, Hkv, T, D).to(dt), src.normal(B, Hkv, T, D).to(dt)) for _ in range(cfg["num_hidden_layers"])]
    return cfg, w, kv, src.lengths(B, T), src.ints(V, B).to(torch.int32)


def _mlp_inputs(case, seed):
    src, dt, h, inter, bits = _Source(seed), DT[case["dtype"]], case["hidden"], case["inter"], case["bits"]
    return dict(gate_up=src.quantised(2 * inter, h, bits, dt), down=src.quantised(h, inter, bits, dt), norm=src.norm(h, dt), h=src.normal(case["rows"], h))


def _attend_inputs(case, seed):
    src, dt, B, D = _Source(seed), DT[case["dtype"]], case["batch"], 128
    L, T, Hq, Hkv = case.get("tokens", 1), case["context"], case["heads"], case["kv_heads"]
    cap = -(-(T + L) // 256) * 256
    norms = (src.norm(D, dt), src.norm(D, dt)) if case["qk_norm"] else (None, None)
    return dict(qkv=src.normal(B * L, (Hq + 2 * Hkv) * D).to(dt), keys=src.normal(B, Hkv, cap, D).to(dt), values=src.normal(B, Hkv, cap, D).to(dt),
                lengths=src.lengths(B, T), q_norm=norms[0], k_norm=norms[1])


def _experts_inputs(case, seed):
    src, dt, W, ff, E = _Source(seed), DT[case["dtype"]], case["width"], case["ff"], case["experts"]
    d = dict(x=src.normal(case["tokens"], W).to(dt), router=src.matrix(E, W, dt), bias=0.1 * src.normal(E),
             gate=[src.matrix(ff, W, dt) for _ in range(E)], up=[src.matrix(ff, W, dt) for _ in range(E)], down=[src.matrix(W, ff, dt) for _ in range(E)])
    if case["shared"]:
        n = case["shared"]
        d["shared"] = (src.matrix(n, W, dt), src.matrix(n, W, dt), src.matrix(W, n, dt))
    return d


def _delta_lens(case):
    """Prompt lengths spread evenly from all of ``tokens`` down to half of them."""
    return [max(1, case["tokens"] - i * case["tokens"] // (2 * case["batch"])) for i in range(case["batch"])]


def _delta_inputs(case, seed):
    src, dt, W, H, G, D = _Source(seed), DT[case["dtype"]], case["width"], case["heads"], case["kv_heads"], case["dim"]
    r = W // 16
    lens = _delta_lens(case)
    return dict(lens=lens, x=src.normal(sum(lens), W).to(dt), q=src.matrix(G * D, W, dt), k=src.matrix(G * D, W, dt), v=src.matrix(H * D, W, dt),
                b=src.matrix(H, W, dt), g1=src.matrix(r, W, dt), g2=src.matrix(H * D, r, dt), a1=src.matrix(r, W, dt), a2=src.matrix(H * D, r, dt),
                o=src.matrix(W, H * D, dt), conv=0.5 * src.normal(2 * G * D + H * D, TAPS), A_log=src.uniform(H) * 3.0 - 2.0,
                dt_bias=src.normal(H * D), norm=1.0 + 0.02 * src.normal(D))


# ---------------------------------------------------------------------------------------------------------------------
# what a program holds before the call
def _linear(parts, bits, group=GROUP):
    w, s, b = parts
    lin = QuantizedLinear(w.shape[1] * 32 // bits, w.shape[0], group, bits)
    lin.set(w, s, b)
    return lin


def _prepare_step(case, seed):
    cfg, w, kv, lengths, ids = _step_inputs(case, seed)
    mod = qwen3 if cfg["model_type"] == "qwen3" else llama
    model = mod.Model(mod.ModelArgs.from_dict(cfg))
    model.load_weights(w, device=DEV)
    B, T = case["batch"], case["context"]
    cache = model.make_cache(B, step=256)
    prepare_cache(cache, B, T + 1, model.dtype, model.device)
    offsets = lengths.tolist()
    for c, (k, v) in zip(cache, kv):
        c.keys[:, :, :T], c.values[:, :, :T] = k, v
        c.offsets_list = offsets
        c.offset = max(offsets)
    session = DecodeSession(model, cache, B, True)
    session.tok.copy_(ids)
    session.run()                       # captures the step
    advance_cache(cache, -1)
    return dict(kind="step", session=session, cache=cache, ids=ids)


def _prepare_mlp(case, seed):
    d = _mlp_inputs(case, seed)
    dt, M, h, inter, bits = DT[case["dtype"]], case["rows"], case["hidden"], case["inter"], case["bits"]
    ws = max(ops.qmm_workspace_bytes(M, 2 * inter, h), ops.qmm_workspace_bytes(M, h, inter), 16)
    return dict(kind="mlp", gate_up=_linear(d["gate_up"], bits), down=_linear(d["down"], bits), norm=d["norm"], h0=d["h"], perm=bits == 4,
                h=torch.empty_like(d["h"]), x=torch.empty((M, h), dtype=dt, device=DEV), act=torch.empty((M, inter), dtype=dt, device=DEV),
                ws=torch.zeros((ws,), dtype=torch.uint8, device=DEV))


def _prepare_attend(case, seed):
    d = _attend_inputs(case, seed)
    B, L, Hq, D = case["batch"], case.get("tokens", 1), case["heads"], 128
    d.update(kind="attend", B=B, L=L, Hq=Hq, Hkv=case["kv_heads"], D=D, q=torch.empty((B * L, Hq * D), dtype=d["qkv"].dtype, device=DEV),
             out=torch.empty((B * L, Hq * D), dtype=d["qkv"].dtype, device=DEV),
             ws=torch.empty((max(ops.attn_workspace_bytes(B, L, Hq, D), 16),), dtype=torch.uint8, device=DEV))
    return d


def _prepare_experts(case, seed):
    d = _experts_inputs(case, seed)
    dt, M, W = DT[case["dtype"]], case["tokens"], case["width"]
    m = RoutedExperts(W, case["experts"], case["top"], case["ff"], "silu", shared_ff=case["shared"])
    m.router.weight, m.router_bias = d["router"], d["bias"]
    m.gate_up = torch.stack([GatedFF.interleave(g, u) for g, u in zip(d["gate"], d["up"])], 0).contiguous()
    m.down = torch.stack(d["down"], 0).contiguous()
    if case["shared"]:
        m.shared.gate_up.weight, m.shared.down.weight = GatedFF.interleave(d["shared"][0], d["shared"][1]).contiguous(), d["shared"][2]
    s = Scratch(torch.device(DEV), M)
    m.reserve(s, dt)
    s.allocate()
    return dict(kind="experts", module=m, scratch=s, x=d["x"], y=torch.empty((M, W), dtype=torch.float32, device=DEV))


def _prepare_delta(case, seed):
    d = _delta_inputs(case, seed)
    dt, W, H, G, D, nb = DT[case["dtype"]], case["width"], case["heads"], case["kv_heads"], case["dim"], case["batch"]
    m = GatedDeltaMixer(W, H, G, D, D, TAPS, DELTA_EPS, channel_decay=True, decay_rank=W // 16, gate_rank=W // 16, gate_act="sigmoid")
    m.in_proj.weight = m.stack_in_proj(d["q"].cpu(), d["k"].cpu(), d["v"].cpu(), d["b"].cpu(), d["g1"].cpu(), d["a1"].cpu()).to(DEV).contiguous()
    m.decay_up.weight, m.gate_up.weight, m.o_proj.weight = d["a2"], d["g2"], d["o"]
    m.conv_w, m.A_log, m.dt_bias, m.norm_w = d["conv"], d["A_log"], d["dt_bias"], d["norm"]
    st = m.new_state(nb)
    st.ensure_capacity(case["tokens"], dt, torch.device(DEV))
    M, i32 = sum(d["lens"]), dict(dtype=torch.int32, device=DEV)
    cu = torch.tensor([0] + torch.tensor(d["lens"]).cumsum(0).tolist(), **i32)
    plan = dict(cu=cu, rows=torch.arange(nb, **i32), nb=nb, lengths=torch.zeros(nb, **i32), max_n=max(d["lens"]), t_row=torch.zeros(M, **i32),
                t_pos=torch.zeros(M, **i32), t_off=torch.zeros(M, **i32))
    ops.ragged_plan(cu, plan["rows"], plan["lengths"], plan["t_row"], plan["t_pos"], plan["t_off"], nb, M)
    s = Scratch(torch.device(DEV), M)
    m.reserve(s, dt)
    s.allocate()
    return dict(kind="delta", module=m, scratch=s, state=st, plan=plan, x=d["x"], y=torch.empty((M, W), dtype=torch.float32, device=DEV))


def prepare(case, seed):
    return {"step": _prepare_step, "mlp": _prepare_mlp, "decode": _prepare_attend, "prompt": _prepare_attend, "experts": _prepare_experts,
            "delta": _prepare_delta}[case["kind"]](case, seed)


# ---------------------------------------------------------------------------------------------------------------------
def run(s):
    if s["kind"] == "step":
        session = s["session"]
        session.tok.copy_(s["ids"])
        session.run()
        advance_cache(s["cache"], -1)       # the next pass takes the same step again
        return {"logits": session.logits}
    if s["kind"] == "mlp":
        s["h"].copy_(s["h0"])
        p = s["perm"]
        ops.rmsnorm(s["h"], s["norm"], EPS, out=s["x"], out_perm=p)
        s["gate_up"](s["x"], EPI_SILU_MUL, out=s["act"], workspace=s["ws"], x_perm=p, y_perm=p)
        s["down"](s["act"], EPI_ADD_RESIDUAL, out=s["h"], workspace=s["ws"], x_perm=p)
        return {"h": s["h"]}
    if s["kind"] == "attend":
        B, L, Hq, Hkv, D = s["B"], s["L"], s["Hq"], s["Hkv"], s["D"]
        ops.rope_kv_append(s["qkv"], s["q"], s["keys"], s["values"], s["lengths"], B, L, Hq, Hkv, D, 500000.0, 1.0, s["q_norm"], s["k_norm"], 1e-6)
        ops.attn(s["q"], s["keys"], s["values"], s["lengths"], s["out"], B, L, Hq, Hkv, D, D ** -0.5, workspace=s["ws"])
        return {"out": s["out"], "keys": s["keys"], "values": s["values"]}
    if s["kind"] == "experts":
        return {"y": s["module"](s["x"], s["y"], s["scratch"])}
    s["module"](s["x"], s["y"], s["state"], s["plan"], s["scratch"], None)
    return {"y": s["y"], "state": s["state"].state, "conv": s["state"].conv}


# ---------------------------------------------------------------------------------------------------------------------
def _qbytes(n, k, bits):
    return n * k * bits / 8 + 2 * n * (k // GROUP) * 2


def work(case):
    kind = case["kind"]
    if kind == "step":
        cfg, B, T = _step_cfg(case), case["batch"], case["context"]
        h, inter, V, L = cfg["hidden_size"], cfg["intermediate_size"], cfg["vocab_size"], cfg["num_hidden_layers"]
        D = cfg.get("head_dim") or h // cfg["num_attention_heads"]
        Hq, Hkv, bits = cfg["num_attention_heads"], cfg["num_key_value_heads"], cfg["quantization"]["bits"]
        mats = [((Hq + 2 * Hkv) * D, h), (h, Hq * D), (2 * inter, h), (h, inter)]
        kept = 0.75 * B * T                                          # mean of the ragged lengths
        weights = sum(_qbytes(n, k, bits) for n, k in mats) * L + _qbytes(V, h, bits)
        macs = sum(n * k for n, k in mats) * L + V * h
        return {"bytes": weights + kept * Hkv * D * 4 * L + B * V * 4, "flops": 2.0 * B * macs + 4.0 * kept * Hq * D * L}
    if kind == "mlp":
        h, inter, M, bits = case["hidden"], case["inter"], case["rows"], case["bits"]
        return {"bytes": _qbytes(2 * inter, h, bits) + _qbytes(h, inter, bits) + M * h * 8, "flops": 6.0 * M * h * inter}
    if kind in ("decode", "prompt"):
        B, L, D, Hq, Hkv = case["batch"], case.get("tokens", 1), 128, case["heads"], case["kv_heads"]
        kept = 0.75 * case["context"]
        pairs = B * (L * kept + L * (L + 1) / 2)
        return {"bytes": B * (kept + 2 * L) * Hkv * D * 4 + 2 * B * L * Hq * D * 2, "flops": 4.0 * pairs * Hq * D}
    if kind == "experts":
        M, W, ff, E, top, n = case["tokens"], case["width"], case["ff"], case["experts"], case["top"], case["shared"]
        hit = E * (1 - (1 - top / E) ** M)                           # experts that at least one token chose
        return {"bytes": hit * 3 * W * ff * 2 + 3 * W * n * 2 + E * W * 2 + M * W * 6, "flops": 6.0 * M * W * (top * ff + n) + 2.0 * M * W * E}
    W, H, G, D = case["width"], case["heads"], case["kv_heads"], case["dim"]
    M, r = sum(_delta_lens(case)), W // 16
    macs = W * (2 * G * D + H * D + H + 2 * r) + 2 * r * H * D + W * H * D
    return {"bytes": macs * 2 + M * W * 6 + case["batch"] * H * D * D * 4, "flops": 2.0 * M * macs + 8.0 * M * H * D * D}


def tolerance(case):
    """About four times what was measured against 64-bit arithmetic: the 16-bit roundings of what travels between the products."""
    half = case["dtype"] == "f16"
    kind = case["kind"]
    if kind == "step":                                   # 5.6e-4 and 4.6e-3
        return {"rel": 2.4e-3 if half else 1.9e-2}
    if kind == "mlp":                                    # 7e-5 and 5.7e-4 (the residual stream is most of the result)
        return {"rel": 3e-4 if half else 2.4e-3}
    if kind in ("decode", "prompt"):                     # 3.5e-4 and 3.5e-3
        return {"rel": 1.4e-3 if half else 1.4e-2}
    if kind == "experts":                                # 1.7e-3; a token at a near tie may take another expert: about 1 / sqrt(tokens)
        return {"rel": 2e-2}
    return {"rel": 7.5e-3}                               # 1.8e-3


# ---------------------------------------------------------------------------------------------------------------------
# the same in 64 bits, plain torch
def _dequantised(parts, bits):
    w, s, b = parts
    shift = torch.arange(0, 32, bits, device=w.device, dtype=torch.int32)
    codes = ((w.unsqueeze(-1) >> shift) & ((1 << bits) - 1)).reshape(w.shape[0], -1, GROUP).double()
    return (codes * s.double().unsqueeze(-1) + b.double().unsqueeze(-1)).reshape(w.shape[0], -1)


def _times(x, parts, bits, rows=16384):
    """x . W^T, the rows of W a block at a time."""
    return torch.cat([x @ _dequantised([t[i:i + rows] for t in parts], bits).t() for i in range(0, parts[0].shape[0], rows)], 1)


def _unit(x, w, eps):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps) * w.double()


def _rope(x, pos, base):
    """x [.., L, D], positions [.., L]: pairs (i, i + D/2)."""
    half = x.shape[-1] // 2
    ang = pos.double().unsqueeze(-1) * torch.pow(torch.tensor(float(base), dtype=torch.float64, device=x.device), -torch.arange(half, device=x.device).double() / half)
    c, s = ang.cos(), ang.sin()
    a, b = x[..., :half], x[..., half:]
    return torch.cat([a * c - b * s, b * c + a * s], -1)


def _attend(qkv, keys, values, lengths, B, L, Hq, Hkv, D, base, wq, wk, eps):
    """qkv [B * L, ..] in 64 bits; keys, values [B, Hkv, cap, D] as stored: outputs and the caches with the new rows."""
    t = qkv.view(B, L, Hq + 2 * Hkv, D).transpose(1, 2)
    q, k, v = t[:, :Hq], t[:, Hq:Hq + Hkv], t[:, Hq + Hkv:]
    if wq is not None:
        q, k = _unit(q, wq, eps), _unit(k, wk, eps)
    pos = lengths.long().unsqueeze(1) + torch.arange(L, device=qkv.device)
    q, k = _rope(q, pos.unsqueeze(1), base), _rope(k, pos.unsqueeze(1), base)
    keys, values = keys.double(), values.double()
    out = torch.empty((B, L, Hq, D), dtype=torch.float64, device=qkv.device)
    for b in range(B):
        n = int(lengths[b])
        keys[b, :, n:n + L], values[b, :, n:n + L] = k[b], v[b]
        kb, vb = keys[b, :, :n + L], values[b, :, :n + L]
        col = torch.arange(n + L, device=qkv.device)
        for i in range(0, L, 512):
            qi = q[b, :, i:i + 512].reshape(Hkv, Hq // Hkv, -1, D)
            m = qi.shape[2]
            sc = torch.einsum("ghld,gtd->ghlt", qi, kb) * D ** -0.5
            sc.masked_fill_(col > (n + i + torch.arange(m, device=qkv.device)).unsqueeze(1), -math.inf)
            out[b, i:i + m] = torch.einsum("ghlt,gtd->lghd", sc.softmax(-1), vb).reshape(m, Hq, D)
    return out.reshape(B * L, Hq * D), keys, values


def _exact_step(case, seed):
    cfg, w, kv, lengths, ids = _step_inputs(case, seed)
    h_, D = cfg["hidden_size"], cfg.get("head_dim") or cfg["hidden_size"] // cfg["num_attention_heads"]
    Hq, Hkv, bits, eps, B = cfg["num_attention_heads"], cfg["num_key_value_heads"], cfg["quantization"]["bits"], cfg["rms_norm_eps"], case["batch"]

    def mat(name):
        return [w[name + "." + leaf] for leaf in ("weight", "scales", "biases")]

    h = _dequantised([t[ids.long()] for t in mat("model.embed_tokens")], bits)
    for i, (k, v) in enumerate(kv):
        p = f"model.layers.{i}."
        x = _unit(h, w[p + "input_layernorm.weight"], eps)
        qkv = torch.cat([_times(x, mat(p + f"self_attn.{n}_proj"), bits) for n in "qkv"], 1)
        pad = torch.zeros((B, Hkv, 1, D), dtype=k.dtype, device=k.device)
        out, _, _ = _attend(qkv, torch.cat([k, pad], 2), torch.cat([v, pad], 2), lengths, B, 1, Hq, Hkv, D, cfg["rope_theta"],
                            w.get(p + "self_attn.q_norm.weight"), w.get(p + "self_attn.k_norm.weight"), eps)
        h = h + _times(out, mat(p + "self_attn.o_proj"), bits)
        x = _unit(h, w[p + "post_attention_layernorm.weight"], eps)
        g, u = _times(x, mat(p + "mlp.gate_proj"), bits), _times(x, mat(p + "mlp.up_proj"), bits)
        h = h + _times(torch.nn.functional.silu(g) * u, mat(p + "mlp.down_proj"), bits)
    return {"logits": _times(_unit(h, w["model.norm.weight"], eps), mat("lm_head"), bits)}


def _exact_mlp(case, seed):
    d, bits, inter = _mlp_inputs(case, seed), case["bits"], case["inter"]
    h = d["h"].double()
    gu = _times(_unit(h, d["norm"], EPS), d["gate_up"], bits)
    return {"h": h + _times(torch.nn.functional.silu(gu[:, :inter]) * gu[:, inter:], d["down"], bits)}


def _exact_attend(case, seed):
    d = _attend_inputs(case, seed)
    out, keys, values = _attend(d["qkv"].double(), d["keys"], d["values"], d["lengths"], case["batch"], case.get("tokens", 1), case["heads"],
                                case["kv_heads"], 128, 500000.0, d["q_norm"], d["k_norm"], 1e-6)
    return {"out": out, "keys": keys, "values": values}


def _exact_experts(case, seed):
    d, top = _experts_inputs(case, seed), case["top"]
    x = d["x"].double()

    def ff(x, g, u, down):
        return (torch.nn.functional.silu(x @ g.double().t()) * (x @ u.double().t())) @ down.double().t()

    val, idx = (x @ d["router"].double().t() + d["bias"].double()).topk(top, -1)
    wts = val.softmax(-1)
    y = ff(x, *d["shared"]) if case["shared"] else torch.zeros_like(x)
    for e in range(case["experts"]):
        tok, k = (idx == e).nonzero(as_tuple=True)
        y.index_add_(0, tok, ff(x[tok], d["gate"][e], d["up"][e], d["down"][e]) * wts[tok, k].unsqueeze(1))
    return {"y": y}


def _exact_delta(case, seed):
    d, H, G, D = _delta_inputs(case, seed), case["heads"], case["kv_heads"], case["dim"]
    F = torch.nn.functional
    x, lens = d["x"].double(), d["lens"]
    nb, n = len(lens), max(lens)
    pre = torch.cat([x @ d[p].double().t() for p in "qkv"], 1)
    C = pre.shape[1]
    beta = (x @ d["b"].double().t()).sigmoid()
    gate = ((x @ d["g1"].double().t()) @ d["g2"].double().t()).sigmoid()
    step = F.softplus((x @ d["a1"].double().t()) @ d["a2"].double().t() + d["dt_bias"].double())
    decay = torch.exp(-d["A_log"].double().exp().view(H, 1) * step.view(-1, H, D))
    # one padded row per sequence: [nb, n, ..]
    start = [sum(lens[:e]) for e in range(nb)]
    take = torch.tensor([[start[e] + min(i, lens[e] - 1) for i in range(n)] for e in range(nb)], device=x.device)
    live = torch.tensor([[i < lens[e] for i in range(n)] for e in range(nb)], device=x.device)
    seq = pre[take]
    past = torch.cat([torch.zeros((nb, TAPS - 1, C), dtype=torch.float64, device=x.device), seq], 1)
    act = F.silu(sum(d["conv"].double()[:, j] * past[:, j:j + n] for j in range(TAPS)))
    q, k = act[..., :G * D].view(nb, n, G, D), act[..., G * D:2 * G * D].view(nb, n, G, D)
    v = act[..., 2 * G * D:].view(nb, n, H, D)
    q = q * torch.rsqrt(q.square().sum(-1, keepdim=True) + 1e-6) * D ** -0.5
    k = k * torch.rsqrt(k.square().sum(-1, keepdim=True) + 1e-6)
    q, k = q.repeat_interleave(H // G, 2), k.repeat_interleave(H // G, 2)
    bt, dc = beta[take], decay[take]
    S = torch.zeros((nb, H, D, D), dtype=torch.float64, device=x.device)
    o = torch.empty((nb, n, H, D), dtype=torch.float64, device=x.device)
    for i in range(n):
        new = S * dc[:, i].unsqueeze(-1)
        u = bt[:, i].unsqueeze(-1) * (v[:, i] - torch.einsum("bhkv,bhk->bhv", new, k[:, i]))
        new = new + k[:, i].unsqueeze(-1) * u.unsqueeze(-2)
        o[:, i] = torch.einsum("bhkv,bhk->bhv", new, q[:, i])
        S = torch.where(live[:, i].view(nb, 1, 1, 1), new, S)
    o = torch.cat([o[e, :lens[e]] for e in range(nb)], 0)
    mix = (_unit(o, d["norm"], DELTA_EPS)).reshape(-1, H * D) * gate
    tail = torch.stack([past[e, lens[e]:lens[e] + TAPS - 1] for e in range(nb)], 0)
    return {"y": mix @ d["o"].double().t(), "state": S, "conv": tail}


def exact(case, seed):
    return {"step": _exact_step, "mlp": _exact_mlp, "decode": _exact_attend, "prompt": _exact_attend, "experts": _exact_experts,
            "delta": _exact_delta}[case["kind"]](case, seed)
