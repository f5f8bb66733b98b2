"""The work that the framework's speed is measured on, through the entry points a user's program calls: NanoChat training steps, the
Laguna mixture of experts, Qwen3.5 prompts and decoding steps, Flux denoising passes.  Widths, depths, batches and lengths come from the
repository's model presets, benchmarks and command lines; ragged lengths and batches in between are generic.

``prepare`` builds models from the seed on the GPU (random weights with the spread of the models' own ``init``), ``run`` is one pass and
``exact`` the same pass in plain torch with 64-bit numbers.
"""
from __future__ import annotations

import math

import torch
import torch.nn.functional as F
from torch.utils.checkpoint import checkpoint

from tyr_b200.models import flux, laguna, qwen35
from tyr_b200.models import nanochat as nc
from tyr_b200.ops import fp4
from tyr_b200.ops import moe as moe_ops
from tyr_b200.train import nanochat_engine as engine
from tyr_b200.utils.graph import GraphedStep

DEV = "cuda"
BF16, F64 = torch.bfloat16, torch.float64


def listed():
    return [
        # a training step of a toy model, as in a first trial run: hundreds of launches of next to no work
        {"name": "train_d4_small", "kind": "train", "depth": 4, "vocab": 4096, "batch": 3, "seq": 250},
        # a medium model with a small device batch and a sequence that is no multiple of a tile
        {"name": "train_d12", "kind": "train", "depth": 12, "vocab": 32768, "batch": 8, "seq": 1000},
        # the headline model and sequence, the device batch of one gradient-accumulation step
        {"name": "train_d20", "kind": "train", "depth": 20, "vocab": 65536, "batch": 8, "seq": 2048},
        # one decoded token through a mixture-of-experts layer (the captured form that a decoding session replays)
        {"name": "moe_1", "kind": "moe", "shape": "s21", "tokens": 1},
        # a batch of 64 decoded tokens through a layer of the benchmark's mixture of experts
        {"name": "moe_64", "kind": "moe", "shape": "bench", "tokens": 64},
        # a prompt of ragged length through a layer of the full-size mixture of experts
        {"name": "moe_prompt", "kind": "moe", "shape": "s21", "tokens": 4000},
        # one user's chat with the smallest preset: a step is a chain of short launches
        {"name": "decode_small_b1", "kind": "decode", "model": "0.8b", "batch": 1, "context": 500},
        # serving many users with the widths of the large preset
        {"name": "decode_large_b32", "kind": "decode", "model": "27b", "batch": 32, "context": 512},
        # time to the first token of a short question to the smallest preset
        {"name": "prompt_small", "kind": "prompt", "model": "0.8b", "batch": 1, "seq": 333},
        # a batch of full prompts at the widths of the large preset
        {"name": "prompt_large", "kind": "prompt", "model": "27b", "batch": 4, "seq": 2048},
        # a denoising pass of a small preview picture
        {"name": "flux_256", "kind": "flux", "batch": 1, "side": 16, "text": 77},
        # a denoising pass of the usual picture: 1024 x 1024 with 512 text tokens
        {"name": "flux_1024", "kind": "flux", "batch": 1, "side": 64, "text": 512},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("train", "moe", "decode", "prompt", "flux"))
    if kind == "train":
        depth = rng.choice((4, 6, 8, 12, 16))
        seq = _log(rng, 100, 2048)
        return {"kind": kind, "depth": depth, "vocab": rng.choice((4096, 16384, 32768)), "batch": _log(rng, 1, max(1, 16384 // seq)), "seq": seq}
    if kind == "moe":
        return {"kind": kind, "shape": rng.choice(("bench", "s21")), "tokens": _log(rng, 1, 8192)}
    if kind == "decode":
        return {"kind": kind, "model": rng.choice(("0.8b", "9b", "27b")), "batch": _log(rng, 1, 40), "context": _log(rng, 20, 640)}
    if kind == "prompt":
        seq = _log(rng, 40, 2048)
        return {"kind": kind, "model": rng.choice(("0.8b", "9b", "27b")), "batch": _log(rng, 1, max(1, 8192 // seq)), "seq": seq}
    side = rng.choice((16, 24, 32, 48, 64))
    return {"kind": kind, "batch": rng.randint(1, max(1, 2048 // (side * side))), "side": side, "text": rng.randint(20, 512)}


# ---- inputs ----------------------------------------------------------------------------------------------------
class _Draws:
    """Random tensors of one seed, on the GPU."""

    def __init__(self, seed):
        self.gen = torch.Generator(device=DEV).manual_seed(seed)

    def normal(self, *shape, std=1.0, dtype=BF16):
        return torch.empty(shape, dtype=dtype, device=DEV).normal_(0.0, std, generator=self.gen)

    def uniform(self, *shape, lo=0.0, hi=1.0, dtype=torch.float32):
        return torch.empty(shape, dtype=dtype, device=DEV).uniform_(lo, hi, generator=self.gen)

    def tokens(self, vocab, *shape):
        return torch.randint(0, vocab, shape, device=DEV, generator=self.gen)


# ---- NanoChat training -------------------------------------------------------------------------------------------
# A trainer in mid-training: matrices that no longer are zero, first and second moments, the learning rates of step 1000.
TRAIN_STEP = 1000


def _train_config(case):
    return nc.depth_config(case["depth"], vocab_size=case["vocab"], max_seq_len=case["seq"])


def _train_inputs(case, seed):
    cfg, r = _train_config(case), _Draws(seed)
    d, V, L = cfg.model_dim, cfg.vocab_size, cfg.n_layer
    f32 = dict(dtype=torch.float32)
    attn = [l for l in range(L) if l != nc.SKIP_ATTN_LAYER]
    w = {"embed": r.normal(V, d, std=0.02, **f32), "smearGate.weight": r.normal(1, 12, std=0.2, **f32),
         "lmHead.weight": r.normal(V, d, std=0.02, **f32), "scalars.values": 1.1 + r.normal(4 * L + 8, std=0.1, **f32)}
    for i in range(cfg.num_value_embeds):
        w[f"valueEmbeds.{i}"] = r.normal(V, d, std=0.02, **f32)
    for l in range(L):
        if l in attn:
            for n in ("wQ", "wK", "wV"):
                w[f"blocks.{l}.attn.{n}"] = r.normal(d, d, std=math.sqrt(3.0 / d), **f32)
            w[f"blocks.{l}.attn.wO"] = r.normal(d, d, std=0.5 / math.sqrt(d), **f32)
        w[f"blocks.{l}.mlp.cFc"] = r.normal(4 * d, d, std=0.02, **f32)
        w[f"blocks.{l}.mlp.cProj"] = r.normal(4 * d, d, std=0.02, **f32)
    shapes = {"embed": (V, d), "value_embeds": (cfg.num_value_embeds, V, d), "lm_head": (V, d), "scalars": (4 * L + 8,)}
    opt = {}
    for k, s in shapes.items():
        size = 1e-3 if k == "scalars" else 2e-5              # of the gradients, so that an update is a fair share of the learning rate
        opt[f"adam.{k}.exp_avg"] = r.normal(*s, std=0.3 * size, **f32)
        opt[f"adam.{k}.exp_avg_sq"] = r.uniform(*s, lo=0.5, hi=2.0).mul_(size * size)
    for k, s in {"attn_w": (len(attn), 4, d, d), "mlp_w": (L, 2, 4 * d, d)}.items():
        opt[f"muon.{k}.momentum"] = r.normal(*s, std=2e-5, **f32)
    opt["muon.smear_gate.momentum"] = r.normal(1, 12, std=1e-3, **f32)
    ids = (r.uniform(case["batch"], case["seq"] + 1, dtype=F64).square_() * V).long().clamp_(0, V - 1)     # frequent tokens and rare ones
    return cfg, w, opt, ids


def _train_prepare(case, seed):
    cfg, w, opt, ids = _train_inputs(case, seed)
    hp = engine.Hyperparameters(device_batch_size=case["batch"], max_seq_len=case["seq"], total_batch_size_tokens=case["batch"] * case["seq"])
    trainer = engine.NanoChatTrainer(cfg, hp, device=DEV, compute_dtype=BF16, seed=0)
    inp, tgt = ids[:, :-1].contiguous(), ids[:, 1:].contiguous()
    for _ in range(3):                              # steps that are behind a trainer in mid-training: the third captures its graph
        trainer.step([(inp, tgt)])
    trainer.params.load_named(w)
    for k in ("embed", "value_embeds", "lm_head", "scalars"):
        opt[f"adam.{k}.step"] = torch.tensor([TRAIN_STEP], dtype=torch.int64)
    trainer.load_optimizer_state_dict(opt)
    trainer.step_index = TRAIN_STEP
    return {"kind": "train", "trainer": trainer, "inp": inp, "tgt": tgt}


def _train_run(s):
    t = s["trainer"]
    out = t.step([(s["inp"], s["tgt"])])
    p = t.params
    # not among the gradients: those of the smear gate and of the per-layer scalars.  Norms follow them, so that what is left of their sums
    # in 16-bit activations is mostly rounding (the updates that are made of them are there all the same).
    grads = {k: p.grad[k] for k in ("embed", "value_embeds", "attn_w", "mlp_w", "lm_head")}
    return {"loss": out.loss, "grads": grads, "params": dict(p.master)}


def _rms(x, eps=1e-6):
    return x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + eps)


def _half_rotary(x, cos, sin):
    """x: [..., S, H, D]; the first half of the channels pairs with the second; cos, sin: [S, D / 2]."""
    a, b = x.chunk(2, -1)
    c, s = cos[:, None], sin[:, None]
    return torch.cat([a * c - b * s, a * s + b * c], -1)


def _causal(q, k, v, scale):
    """[B, S, H, D] with fewer key heads than query heads allowed; a few rows of the batch at a time."""
    B, S, H, _ = q.shape
    rep = H // k.shape[2]
    mask = torch.ones(S, S, dtype=torch.bool, device=q.device).triu(1)
    step = max(1, int(2 ** 28 // max(1, H * S * S)))

    def rows(q, k, v):
        p = torch.einsum("bihd,bjhd->bhij", q, k.repeat_interleave(rep, 2)) * scale
        return torch.einsum("bhij,bjhd->bihd", p.masked_fill(mask, -math.inf).softmax(-1), v.repeat_interleave(rep, 2))
    call = (lambda *a: checkpoint(rows, *a, use_reentrant=False)) if q.requires_grad else rows
    return torch.cat([call(q[i:i + step], k[i:i + step], v[i:i + step]) for i in range(0, B, step)])


def _orthogonal(u):
    """Muon's five Newton-Schulz steps on matrices of unit norm."""
    a, b, c = 3.4445, -4.7750, 2.0315
    x = u / (u.square().sum((-2, -1), keepdim=True).sqrt() + 1e-7)
    tall = x.shape[-2] > x.shape[-1]
    x = x.mT if tall else x
    for _ in range(5):
        s = x @ x.mT
        x = a * x + (b * s + c * s @ s) @ x
    return x.mT if tall else x


def _train_exact(case, seed):
    if case["depth"] * 64 * case["batch"] * case["seq"] > 3.2e7:
        return None
    cfg, w, opt, ids = _train_inputs(case, seed)
    d, V, L, H, D, T = cfg.model_dim, cfg.vocab_size, cfg.n_layer, cfg.n_head, cfg.head_dim, case["seq"]
    # activations and products use 16-bit copies of the weights; scalars and the smear gate stay as they are
    p = {k: (v if k in ("scalars.values", "smearGate.weight") else v.to(BF16)).to(F64).requires_grad_(True) for k, v in w.items()}
    inp, tgt = ids[:, :-1], ids[:, 1:]
    ang = torch.arange(T, device=DEV, dtype=F64)[:, None] * (cfg.rope_base ** -(torch.arange(0, D, 2, device=DEV, dtype=F64) / D))
    cos, sin = ang.cos(), ang.sin()
    sig = torch.sigmoid(p["scalars.values"])
    tok = F.embedding(inp, p["embed"])
    x0 = _rms(tok * (1 + torch.sigmoid(F.linear(tok[..., :12], p["smearGate.weight"]))))
    span = min(cfg.num_value_embeds, L)

    def layer(l, x, skip):
        lam = sig[4 * l:4 * l + 4]
        x = lam[0] * x + lam[1] * x0
        held = x
        if l != nc.SKIP_ATTN_LAYER:
            n = _rms(x)
            q, k, v = (F.linear(n, p[f"blocks.{l}.attn.{m}"]) for m in ("wQ", "wK", "wV"))
            vi = l if l < span else l - (L - span) if l >= L - span else None
            if vi is not None:
                v = (1 - sig[4 * L]) * v + sig[4 * L] * F.embedding(inp, p[f"valueEmbeds.{vi}"])
            q, k, v = (t.unflatten(-1, (H, D)) for t in (q, k, v))
            q, k = _rms(_half_rotary(q, cos, sin)), _rms(_half_rotary(k, cos, sin))
            x = x + lam[2] * F.linear(_causal(q, k, v, D ** -0.5).flatten(-2), p[f"blocks.{l}.attn.wO"])
        elif skip is not None:
            x = x + sig[4 * L + 1] * skip
        h = F.linear(_rms(x), p[f"blocks.{l}.mlp.cFc"]).relu().square()
        return x + lam[3] * (h @ p[f"blocks.{l}.mlp.cProj"]), held

    x, skip = x0, None
    for l in range(L):
        x, held = checkpoint(layer, l, x, skip, use_reentrant=False)
        skip = held if l == nc.SKIP_SOURCE_LAYER else skip
    x = _rms(sig[4 * L + 2] * x).reshape(-1, d)

    def entropy(x, t):
        return F.cross_entropy(torch.tanh(F.linear(x, p["lmHead.weight"]) / cfg.softcap_value) * cfg.softcap_value, t, reduction="sum")
    loss = sum(checkpoint(entropy, a, b, use_reentrant=False) for a, b in zip(x.split(2048), tgt.reshape(-1).split(2048))) / tgt.numel()
    loss.backward()
    g = {k: v.grad if v.grad is not None else torch.zeros_like(v) for k, v in p.items()}
    attn = [l for l in range(L) if l != nc.SKIP_ATTN_LAYER]
    grouped = lambda t: {"embed": t["embed"], "smear_gate": t["smearGate.weight"],
                         "value_embeds": torch.stack([t[f"valueEmbeds.{i}"] for i in range(cfg.num_value_embeds)]),
                         "attn_w": torch.stack([torch.stack([t[f"blocks.{l}.attn.{n}"] for n in ("wQ", "wK", "wV", "wO")]) for l in attn]),
                         "mlp_w": torch.stack([torch.stack([t[f"blocks.{l}.mlp.{n}"] for n in ("cFc", "cProj")]) for l in range(L)]),
                         "lm_head": t["lmHead.weight"], "scalars": t["scalars.values"]}
    with torch.no_grad():
        del p
        grads, new = grouped(g), {}
        for k, m in grouped({k: v.to(F64) for k, v in w.items()}).items():
            batch = math.sqrt(case["batch"] * T / 524288.0)
            if f"adam.{k}.exp_avg" in opt:
                a = 0.8 * opt[f"adam.{k}.exp_avg"].to(F64) + 0.2 * grads[k]
                b = 0.95 * opt[f"adam.{k}.exp_avg_sq"].to(F64) + 0.05 * grads[k].square()
                t = TRAIN_STEP + 1
                lr = (0.3 if "embed" in k else 0.004) * batch * (d / 768.0) ** -0.5
                new[k] = m - lr * (a / (1 - 0.8 ** t)) / ((b / (1 - 0.95 ** t)).sqrt() + 1e-10)
            else:
                a = 0.95 * opt[f"muon.{k}.momentum"].to(F64) + 0.05 * grads[k]
                tall = math.sqrt(m.shape[-2] / m.shape[-1]) if m.shape[-2] > m.shape[-1] else 1.0
                new[k] = m - 0.02 * batch * tall * _orthogonal(0.05 * grads[k] + 0.95 * a)
        return {"loss": loss.detach(), "grads": {k: grads[k] for k in ("embed", "value_embeds", "attn_w", "mlp_w", "lm_head")},
                "params": {k: new[k] for k in ("embed", "smear_gate", "value_embeds", "attn_w", "mlp_w", "lm_head", "scalars")}}


def _train_work(case):
    cfg = _train_config(case)
    d, V, L, N = cfg.model_dim, cfg.vocab_size, cfg.n_layer, case["batch"] * case["seq"]
    La = L - (L > nc.SKIP_ATTN_LAYER)
    matrices = La * 4 * d * d + L * 8 * d * d
    tables = (2 + cfg.num_value_embeds) * V * d
    attention = 3.5 * 2 * case["batch"] * case["seq"] ** 2 * d * La           # causal: half of the four products, and of the backward's ten
    muon = 5 * (La * 4 * 6 * d ** 3 + L * 2 * (2 * 2 * d * d * 4 * d + 2 * d ** 3))
    # masters, moments read and written, gradients and 16-bit copies written
    return {"flops": 6.0 * N * (matrices + V * d) + attention + muon, "bytes": 22.0 * matrices + 30.0 * tables + 16.0 * N}


# ---- Laguna mixture of experts -----------------------------------------------------------------------------------
MOE = {"s21": laguna.LagunaConfig(), "bench": laguna.LagunaConfig(hidden_size=2048, num_experts=64, num_experts_per_tok=8, moe_intermediate_size=768,
                                                                  shared_expert_intermediate_size=768)}
E2M1 = (0.0, 0.5, 1.0, 1.5, 2.0, 3.0, 4.0, 6.0)


def _e4m3(x):
    return x.float().clamp(max=448.0).to(torch.float8_e4m3fn)


def _bank(r, E, rows, cols):
    """Gaussian matrices in NVFP4: (codes of 4 bits in pairs, a scale per 16 numbers, a factor per matrix)."""
    packed = torch.empty((E, rows, cols // 2), dtype=torch.uint8, device=DEV)
    scales = torch.empty((E, rows, cols // 16), dtype=torch.float8_e4m3fn, device=DEV)
    factor = torch.empty(E, dtype=torch.float32, device=DEV)
    mids = torch.tensor([0.25, 0.75, 1.25, 1.75, 2.5, 3.5, 5.0], device=DEV)
    for e in range(0, E, 16):
        w = r.normal(min(16, E - e), rows, cols, std=cols ** -0.5, dtype=torch.float32)
        f = 2688.0 / w.abs().amax((1, 2))
        blocks = w.unflatten(-1, (-1, 16)) * f[:, None, None, None]
        s = _e4m3(blocks.abs().amax(-1) / 6.0)
        q = blocks / s.float().clamp_min(2.0 ** -9)[..., None]
        codes = (torch.bucketize(q.abs(), mids, out_int32=True) + 8 * (q < 0)).to(torch.uint8).flatten(-2)
        packed[e:e + 16], scales[e:e + 16], factor[e:e + 16] = codes[..., 0::2] | codes[..., 1::2] << 4, s, f
    return packed, scales, factor


def _decoded(bank, e):
    packed, scales, factor = (t[e] for t in bank)
    lut = torch.tensor(E2M1 + tuple(-v for v in E2M1), device=DEV, dtype=F64)
    v = torch.stack([lut[(packed & 15).long()], lut[(packed >> 4).long()]], -1).flatten(-2)
    return v * (scales.to(F64) / factor.to(F64)).repeat_interleave(16, -1)


def _moe_inputs(case, seed):
    cfg, r = MOE[case["shape"]], _Draws(seed)
    E, h, mi, si = cfg.num_experts, cfg.hidden_size, cfg.moe_intermediate_size, cfg.shared_expert_intermediate_size
    router = r.normal(E, h, std=h ** -0.5, dtype=torch.float32)
    bias = r.normal(E, std=0.02, dtype=torch.float32)
    shared = r.normal(si, h, std=h ** -0.5), r.normal(si, h, std=h ** -0.5), r.normal(h, si, std=si ** -0.5)
    banks = _bank(r, E, mi, h), _bank(r, E, mi, h), _bank(r, E, h, mi)
    return cfg, router, bias, shared, banks, r.normal(case["tokens"], h)


def _moe_prepare(case, seed):
    getattr(fp4, "_prepared", {}).clear()         # banks of an earlier state may have lain at the same addresses
    cfg, router, bias, shared, banks, x = _moe_inputs(case, seed)
    experts = moe_ops.PackedExperts(*(t for b in banks for t in b))
    block = laguna.SparseMoeBlock(laguna.Router(router, bias), experts, *shared)
    with torch.no_grad():
        layer = lambda x2: laguna.moe_forward(cfg, block, x2)
        if case["tokens"] <= 128:                   # decode-sized: a session captures its step and replays it
            layer = GraphedStep(layer, (x,))
        layout = fp4.prepared(experts)              # laid out once, kept as long as the layer
    return {"kind": "moe", "layer": layer, "x": x, "keep": (block, layout)}


@torch.no_grad()
def _moe_run(s):
    return s["layer"](s["x"])


def _nvfp4(x, row_scale):
    """x as the tensor core's operand: e2m1 numbers with a UE4M3 scale per 16, and a factor per row."""
    g = x.abs().amax(1, keepdim=True) / 2688.0 if row_scale else torch.ones(x.shape[0], 1, device=DEV, dtype=F64)
    b = x.unflatten(-1, (-1, 16))
    s = (_e4m3(b.abs().amax(-1) / g / 6.0).to(F64) * g)[..., None]
    q = torch.where(s > 0, b / s, torch.zeros_like(b))
    grid = torch.tensor(E2M1, device=DEV, dtype=F64)
    mids = (grid[1:] + grid[:-1]) / 2
    low = torch.bucketize(q.abs(), mids)                        # a tie goes to the lower code ...
    tie = (low < 7) & (q.abs() == mids[low.clamp(max=6)]) & (low % 2 == 1)
    return (torch.sign(q) * grid[low + tie] * s).flatten(-2)      # ... unless the upper one is even


def _moe_exact(case, seed):
    cfg, router, bias, shared, banks, x = _moe_inputs(case, seed)
    x, k, T = x.to(F64), cfg.num_experts_per_tok, case["tokens"]
    scores = torch.sigmoid(x @ router.to(F64).T)
    ids = torch.argsort(scores + bias.to(F64), dim=-1, descending=True, stable=True)[:, :k]
    w = scores.gather(1, ids)
    w = w / w.sum(-1, keepdim=True) * cfg.moe_routed_scaling_factor
    g, u, dn = (t.to(F64) for t in shared)
    out = (F.silu(x @ g.T) * (x @ u.T)) @ dn.T
    # more than two pairs per expert take the FP4 tensor cores, whose operands are FP4 on both sides; fewer stream the weights
    tensor_core = T * k > 2 * cfg.num_experts
    xq = _nvfp4(x, True) if tensor_core else x
    for e in ids.unique().tolist():
        t, slot = torch.nonzero(ids == e, as_tuple=True)
        h = F.silu(xq[t] @ _decoded(banks[0], e).T) * (xq[t] @ _decoded(banks[1], e).T)
        h = _nvfp4(h, False) if tensor_core else h
        out.index_add_(0, t, (h @ _decoded(banks[2], e).T) * w[t, slot, None])
    return out


def _moe_work(case):
    cfg, T = MOE[case["shape"]], case["tokens"]
    E, k, h, mi, si = cfg.num_experts, cfg.num_experts_per_tok, cfg.hidden_size, cfg.moe_intermediate_size, cfg.shared_expert_intermediate_size
    active = E * (1 - (1 - k / E) ** T)
    return {"flops": 6.0 * T * h * (k * mi + si) + 2.0 * T * E * h, "bytes": active * 3 * h * mi * 0.5625 + 6.0 * h * si + 4.0 * E * h + 4.0 * T * h}


# ---- Qwen3.5 -----------------------------------------------------------------------------------------------------
def _qwen_config(name):
    if name == "0.8b":
        return qwen35.Qwen35Config.qwen35_0_8b()
    cfg = {"9b": qwen35.Qwen35Config.qwen35_9b, "27b": qwen35.Qwen35Config.qwen35_27b}[name]()
    return qwen35.Qwen35Config(**{f: getattr(cfg, f) for f in ("vocab_size", "hidden_size", "intermediate_size", "num_attention_heads",
                                                               "num_key_value_heads", "linear_num_value_heads")}, num_hidden_layers=8)


STEPS = 64                 # decoded tokens after which a session starts over behind its context


def _qwen_inputs(case, seed):
    cfg, r = _qwen_config(case["model"]), _Draws(seed)
    h, D, H, Hkv, I = cfg.hidden_size, cfg.head_dim, cfg.num_attention_heads, cfg.num_key_value_heads, cfg.intermediate_size
    Hv, cd, vd, K, dv = cfg.linear_num_value_heads, cfg.linear_conv_dim, cfg.linear_value_dim, cfg.linear_conv_kernel_dim, cfg.linear_value_head_dim
    mat = lambda n, k, gain=1.0: r.normal(n, k, std=gain * k ** -0.5)
    small = (2 * cfg.num_hidden_layers) ** -0.5        # what a layer adds to the stream, as deep models are initialised and trained
    layers = []
    for i in range(cfg.num_hidden_layers):
        if cfg.is_full(i):
            m = {"q": mat(2 * H * D, h), "k": mat(Hkv * D, h), "v": mat(Hkv * D, h), "o": mat(h, H * D, small), "qn": r.normal(D, std=0.1), "kn": r.normal(D, std=0.1)}
        else:
            m = {"qkv": mat(cd, h), "z": mat(vd, h), "b": mat(Hv, h), "a": mat(Hv, h), "conv": mat(cd, K).unsqueeze(1), "bias": r.normal(cd, std=0.05),
                 # time steps between 0.001 and 0.1, as such layers start out: a state keeps some ten to a thousand tokens
                 "dt": torch.log(torch.expm1(torch.exp(r.uniform(Hv, lo=math.log(1e-3), hi=math.log(0.1))))),
                 "alog": torch.log(r.uniform(Hv, lo=1.0, hi=16.0)), "norm": 1 + r.normal(dv, std=0.1), "o": mat(h, vd, small)}
        m.update(n1=r.normal(h, std=0.1), n2=r.normal(h, std=0.1), gate=mat(I, h), up=mat(I, h), down=mat(h, I, small))
        layers.append(m)
    emb = r.normal(cfg.vocab_size, h)
    head = emb if cfg.tie_word_embeddings else mat(cfg.vocab_size, h)
    final = r.normal(h, std=0.1)
    rows = case["seq"] if case["kind"] == "prompt" else case["context"] + 1
    return cfg, layers, emb, head, final, r.tokens(cfg.vocab_size, case["batch"], rows)


def _qwen_prepare(case, seed):
    cfg, layers, emb, head, final, ids = _qwen_inputs(case, seed)
    made = []
    for m in layers:
        mixer = (qwen35.Attention(m["q"], m["k"], m["v"], m["o"], m["qn"], m["kn"]) if "q" in m else
                 qwen35.GatedDeltaNet(m["qkv"], m["z"], m["b"], m["a"], m["conv"], m["bias"], m["dt"], m["alog"], m["norm"], m["o"]))
        made.append(qwen35.Layer(m["n1"], mixer, m["n2"], qwen35.MLP(m["gate"], m["up"], m["down"])))
    model = qwen35.Qwen35ForCausalLM(cfg, emb, made, final, head, cfg.tie_word_embeddings)
    if case["kind"] == "prompt":
        return {"kind": "prompt", "model": model, "ids": ids}
    session = qwen35.HybridCache(model, case["batch"], case["context"] + STEPS)
    with torch.no_grad():
        session.prefill(ids[:, :-1])
    return {"kind": "decode", "session": session, "token": ids[:, -1].contiguous(), "context": case["context"]}


@torch.no_grad()
def _prompt_run(s):
    return qwen35.HybridCache(s["model"], s["ids"].shape[0], s["ids"].shape[1] + STEPS).prefill(s["ids"])


@torch.no_grad()
def _decode_run(s):
    session = s["session"]
    if session.pos >= session.max_len:             # no room: go on behind the context, over the tokens decoded before
        session.pos = s["context"]
        session.lengths = [s["context"]] * session.batch
        for c in session.kv:
            if c is not None:
                c.length = s["context"]
        session.pos_t.fill_(s["context"])
    return session.step(s["token"])


def _qwen_exact(case, seed):
    cfg = _qwen_config(case["model"])
    B, S = case["batch"], case["seq"] if case["kind"] == "prompt" else case["context"] + 1
    if B * S * cfg.hidden_size > 4.5e7 * (2.5 if cfg.num_hidden_layers == 8 else 1):
        return None
    cfg, layers, emb, head, final, ids = _qwen_inputs(case, seed)
    D, H, Hkv, half, eps = cfg.head_dim, cfg.num_attention_heads, cfg.num_key_value_heads, cfg.half_rotary_dim, cfg.rms_norm_eps
    Hk, Hv, dk, dv, K = cfg.linear_num_key_heads, cfg.linear_num_value_heads, cfg.linear_key_head_dim, cfg.linear_value_head_dim, cfg.linear_conv_kernel_dim
    ang = torch.arange(S, device=DEV, dtype=F64)[:, None] * (cfg.rope_theta ** -(torch.arange(half, device=DEV, dtype=F64) / half))
    cos, sin = ang.cos(), ang.sin()
    lin = lambda x, w: F.linear(x, w.to(F64))
    norm = lambda x, w: _rms(x, eps) * (1 + w.to(F64))
    turn = lambda x: torch.cat([_half_rotary(x[..., :2 * half], cos, sin), x[..., 2 * half:]], -1)
    unit = lambda x: x * torch.rsqrt(x.square().sum(-1, keepdim=True) + 1e-6)
    with torch.no_grad():
        x = F.embedding(ids, emb).to(F64)
        for m in layers:
            n = norm(x, m["n1"])
            if "q" in m:
                q, gate = lin(n, m["q"]).unflatten(-1, (H, 2 * D)).chunk(2, -1)
                k, v = lin(n, m["k"]).unflatten(-1, (Hkv, D)), lin(n, m["v"]).unflatten(-1, (Hkv, D))
                o = _causal(turn(norm(q, m["qn"])), turn(norm(k, m["kn"])), v, D ** -0.5)
                y = lin((o * torch.sigmoid(gate)).flatten(-2), m["o"])
            else:
                c = F.pad(lin(n, m["qkv"]), (0, 0, K - 1, 0))
                c = F.silu(sum(c[:, t:t + S] * m["conv"][:, 0, t].to(F64) for t in range(K)) + m["bias"].to(F64))
                q, k, v = c.split((Hk * dk, Hk * dk, Hv * dv), -1)
                q, k = (unit(t.unflatten(-1, (Hk, dk))).repeat_interleave(Hv // Hk, 2) for t in (q, k))
                q, v, beta = q * dk ** -0.5, v.unflatten(-1, (Hv, dv)), torch.sigmoid(lin(n, m["b"]))
                decay = torch.exp(-F.softplus(lin(n, m["a"]) + m["dt"].to(F64)) * m["alog"].to(F64).exp())
                state, o = torch.zeros(B * Hv, dk, dv, device=DEV, dtype=F64), torch.empty_like(v)
                flat = lambda t, i: t[:, i].reshape(B * Hv, 1, -1)
                for i in range(S):
                    state.mul_(flat(decay, i))
                    d = (flat(v, i) - flat(k, i) @ state) * flat(beta, i)
                    state.baddbmm_(flat(k, i).mT, d)
                    o[:, i] = (flat(q, i) @ state).reshape(B, Hv, dv)
                o = _rms(o, eps) * m["norm"].to(F64) * F.silu(lin(n, m["z"])).unflatten(-1, (Hv, dv))
                y = lin(o.flatten(-2), m["o"])
            x = x + y
            n = norm(x, m["n2"])
            x = x + lin(F.silu(lin(n, m["gate"])) * lin(n, m["up"]), m["down"])
        x = norm(x[:, -1], final)
        return torch.cat([lin(x, w) for w in head.split(32768)], -1)


def _qwen_work(case):
    cfg = _qwen_config(case["model"])
    B, S = case["batch"], case["seq"] if case["kind"] == "prompt" else 1
    context = 0 if case["kind"] == "prompt" else case["context"]
    h, D, H, Hkv = cfg.hidden_size, cfg.head_dim, cfg.num_attention_heads, cfg.num_key_value_heads
    full = sum(cfg.is_full(i) for i in range(cfg.num_hidden_layers))
    linear = cfg.num_hidden_layers - full
    weights = (full * (3 * H * D + 2 * Hkv * D) * h + linear * (cfg.linear_conv_dim + 2 * cfg.linear_value_dim + 2 * cfg.linear_num_value_heads) * h
               + cfg.num_hidden_layers * 3 * h * cfg.intermediate_size)
    pairs = B * S * (S + 1) / 2 + B * S * context
    state = linear * B * cfg.linear_num_value_heads * cfg.linear_key_head_dim * cfg.linear_value_head_dim
    flops = 2.0 * B * S * weights + 2.0 * B * h * cfg.vocab_size + full * 4.0 * pairs * H * D + 8.0 * S * state
    stores = full * B * (S + context) * 2 * Hkv * D * 2
    return {"flops": flops, "bytes": 2.0 * weights + 2.0 * h * cfg.vocab_size + stores + (8.0 if context else 4.0) * state + 2.0 * B * cfg.vocab_size}


# ---- Flux --------------------------------------------------------------------------------------------------------
def _flux_inputs(case, seed):
    cfg, r = flux.FluxConfig.klein4b(), _Draws(seed)
    h, M, D = cfg.hidden_size, cfg.mlp_hidden_dim, cfg.head_dim
    mat = lambda n, k: r.normal(n, k, std=k ** -0.5)
    gain = lambda: 1 + r.normal(D, std=0.1)
    w = {"img_in": mat(h, cfg.in_channels), "txt_in": mat(h, cfg.context_in_dim), "t1": mat(h, cfg.time_dim), "t2": mat(h, h), "mod_img": mat(6 * h, h),
         "mod_txt": mat(6 * h, h), "mod": mat(3 * h, h), "out": mat(cfg.in_channels, h), "mod_out": mat(2 * h, h)}
    w["double"] = [{s: {"qkv": mat(3 * h, h), "qn": gain(), "kn": gain(), "proj": mat(h, h), "w1": mat(2 * M, h), "w2": mat(h, M)} for s in ("img", "txt")}
                   for _ in range(cfg.num_double_layers)]
    w["single"] = [{"l1": mat(3 * h + 2 * M, h), "l2": mat(h, h + M), "qn": gain(), "kn": gain()} for _ in range(cfg.num_single_layers)]
    B, side, St = case["batch"], case["side"], case["text"]
    img, txt, t = r.normal(B, side * side, cfg.in_channels), r.normal(B, St, cfg.context_in_dim), r.uniform(B, lo=0.05, hi=1.0)
    img_ids, txt_ids = flux.compute_image_position_ids(side, side, DEV), flux.compute_text_position_ids(St, DEV)
    return cfg, w, (img, txt, t, img_ids.expand(B, -1, -1).contiguous(), txt_ids.expand(B, -1, -1).contiguous())


def _flux_prepare(case, seed):
    cfg, w, inputs = _flux_inputs(case, seed)
    attn = lambda b: flux.SelfAttention(b["qkv"], flux.QKNorm(b["qn"], b["kn"]), b["proj"])
    mlp = lambda b: flux.SwiGLUMLP(b["w1"], b["w2"])
    doubles = [flux.DoubleStreamBlock(attn(b["img"]), mlp(b["img"]), attn(b["txt"]), mlp(b["txt"])) for b in w["double"]]
    singles = [flux.SingleStreamBlock(b["l1"], b["l2"], flux.QKNorm(b["qn"], b["kn"])) for b in w["single"]]
    model = flux.FluxModel(cfg, w["img_in"], w["txt_in"], w["t1"], w["t2"], doubles, singles, w["mod_img"], w["mod_txt"], w["mod"], w["out"], w["mod_out"])
    return {"kind": "flux", "model": model, "inputs": inputs}


@torch.no_grad()
def _flux_run(s):
    return flux.forward(s["model"], *s["inputs"])


def _flux_exact(case, seed):
    cfg, w, (img, txt, t, img_ids, txt_ids) = _flux_inputs(case, seed)
    H, D, h, M = cfg.num_heads, cfg.head_dim, cfg.hidden_size, cfg.mlp_hidden_dim
    lin = lambda x, m: F.linear(x, m.to(F64))

    def angles(ids):
        om = [cfg.theta ** -(torch.arange(n, device=DEV, dtype=F64) / n) for n in cfg.half_axes_dims]
        return torch.cat([ids[..., a, None].to(F64) * o for a, o in enumerate(om)], -1)[:, :, None]

    def heads(x, b, ang):
        q, k, v = x.unflatten(-1, (3, H, D)).unbind(2)
        out = []
        for y, g in ((q, b["qn"]), (k, b["kn"])):
            y0, y1 = (_rms(y) * g.to(F64)).unflatten(-1, (D // 2, 2)).unbind(-1)
            out.append(torch.stack([y0 * ang.cos() - y1 * ang.sin(), y0 * ang.sin() + y1 * ang.cos()], -1).flatten(-2))
        return (*out, v)

    def attend(q, k, v):
        each = [(torch.einsum("bid,bjd->bij", q[:, :, n], k[:, :, n]) * D ** -0.5).softmax(-1) @ v[:, :, n] for n in range(H)]
        return torch.cat(each, -1)

    norm = lambda x, shift, scale: F.layer_norm(x, (h,), eps=1e-6) * (1 + scale[:, None]) + shift[:, None]
    glu = lambda x: F.silu(x[..., :M]) * x[..., M:]
    with torch.no_grad():
        half = cfg.time_dim // 2
        ang = t.to(F64)[:, None] * 1000.0 * torch.exp(-math.log(10000.0) * torch.arange(half, device=DEV, dtype=F64) / half)
        vec = F.silu(lin(F.silu(lin(torch.cat([ang.cos(), ang.sin()], -1), w["t1"])), w["t2"]))
        mods = {s: lin(vec, w["mod_" + s]).unflatten(-1, (6, h)).unbind(1) for s in ("img", "txt")}
        x = {"img": lin(img.to(F64), w["img_in"]), "txt": lin(txt.to(F64), w["txt_in"])}
        pe, St = {"img": angles(img_ids), "txt": angles(txt_ids)}, txt.shape[1]
        for b in w["double"]:
            parts = [heads(lin(norm(x[s], *mods[s][:2]), b[s]["qkv"]), b[s], pe[s]) for s in ("txt", "img")]
            o = attend(*(torch.cat(p, 1) for p in zip(*parts)))
            for s, a in (("txt", o[:, :St]), ("img", o[:, St:])):
                m = mods[s]
                x[s] = x[s] + m[2][:, None] * lin(a, b[s]["proj"])
                x[s] = x[s] + m[5][:, None] * lin(glu(lin(norm(x[s], *m[3:5]), b[s]["w1"])), b[s]["w2"])
        x, pe = torch.cat([x["txt"], x["img"]], 1), torch.cat([pe["txt"], pe["img"]], 1)
        m = lin(vec, w["mod"]).unflatten(-1, (3, h)).unbind(1)
        for b in w["single"]:
            y = lin(norm(x, *m[:2]), b["l1"])
            o = attend(*heads(y[..., :3 * h], b, pe))
            x = x + m[2][:, None] * lin(torch.cat([o, glu(y[..., 3 * h:])], -1), b["l2"])
        shift, scale = lin(vec, w["mod_out"]).chunk(2, -1)
        return lin(norm(x[:, St:], shift, scale), w["out"])


def _flux_work(case):
    cfg = flux.FluxConfig.klein4b()
    h, M, B, Si, St = cfg.hidden_size, cfg.mlp_hidden_dim, case["batch"], case["side"] ** 2, case["text"]
    block = 4 * h * h + 3 * h * M
    ends = h * (2 * cfg.in_channels + cfg.context_in_dim + cfg.time_dim) + 18 * h * h
    flops = 2.0 * B * (Si + St) * block * (cfg.num_double_layers + cfg.num_single_layers) + 2.0 * B * h * (2 * Si * cfg.in_channels + St * cfg.context_in_dim)
    flops += 4.0 * B * (Si + St) ** 2 * h * (cfg.num_double_layers + cfg.num_single_layers)
    weights = block * (2 * cfg.num_double_layers + cfg.num_single_layers) + ends
    return {"flops": flops, "bytes": 2.0 * weights + 2.0 * B * (2 * Si * cfg.in_channels + St * cfg.context_in_dim)}


# ---- what is called from outside ---------------------------------------------------------------------------------
PREPARE = {"train": _train_prepare, "moe": _moe_prepare, "decode": _qwen_prepare, "prompt": _qwen_prepare, "flux": _flux_prepare}
RUN = {"train": _train_run, "moe": _moe_run, "decode": _decode_run, "prompt": _prompt_run, "flux": _flux_run}
EXACT = {"train": _train_exact, "moe": _moe_exact, "decode": _qwen_exact, "prompt": _qwen_exact, "flux": _flux_exact}
WORK = {"train": _train_work, "moe": _moe_work, "decode": _qwen_work, "prompt": _qwen_work, "flux": _flux_work}


def prepare(case, seed):
    return PREPARE[case["kind"]](case, seed)


def run(state):
    return RUN[state["kind"]](state)


def exact(case, seed):
    return EXACT[case["kind"]](case, seed)


def work(case):
    return WORK[case["kind"]](case)


def tolerance(case):
    """Measured against ``exact``: gradients are 0.2 to 0.8 % off (single entries of frequent tokens' rows much more), logits 0.8 to 1.4 %, velocities
    1.1 %, and the mixture of experts 2.6 %, where a sum in another order moves numbers across the steps of 4 bits."""
    return {"rel": 0.03, "max": 0.99 if case["kind"] == "train" else 0.5}
