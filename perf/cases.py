"""The work that fine-tuning with this framework consists of, as cases that can be timed and compared.

Each case is one pass through a public entry point: an operator of ``chronicals_b200.ops``, a block of
``chronicals_b200.models.decoder``, an optimizer step, or a whole model.  Shapes are those of the package's
architecture presets; token counts and document lengths are what packed micro-batches look like.
"""
from __future__ import annotations

import dataclasses
import math

import torch

from chronicals_b200 import ops
from chronicals_b200.config.config import ChronicalsConfig
from chronicals_b200.models.decoder import MLP, Attention, CausalLM, FusedLinear
from chronicals_b200.ops import ref
from chronicals_b200.optimizers.fused_adamw import FusedAdamW
from chronicals_b200.utils.fp8_deepseek import convert_model_to_fp8

DEV = "cuda"
BF = torch.bfloat16
IGNORE = -100
PRESETS = ("qwen2.5-0.5b", "qwen2.5-1.5b", "llama-1b", "deepseek-mini", "qwen2.5-7b", "qwen2.5-14b", "tiny-qwen2")

# 27 documents of log-normal lengths, as an instruction data set packs into one micro-batch of 8192 tokens
DOCS_8K = "1024,83,411,97,733,260,1544,61,190,322,35,508,148,91,287,604,212,77,119,451,46,163,205,98,233,144,46"


def listed():
    return [
        # the smallest call: scoring two short prompts with a tiny model, no gradients; launches and latency
        {"name": "eval_tiny", "kind": "model", "arch": "tiny-qwen2", "layers": 4, "vocab": 32000, "lens": "61,97", "train": False},
        # a whole micro-batch of ragged packed documents, forward and backward, through two full decoder layers, the
        # embedding and the fused loss (which dominates a step is seen better in the single cases below)
        {"name": "model_train_0.5b", "kind": "model", "arch": "qwen2.5-0.5b", "layers": 2, "vocab": 32000,
         "lens": "1024,711,83,1340,260,97,508,73", "train": True},
        # the norm in front of every block of a 14B model, with the residual gradient folded in
        {"name": "norm_14b", "kind": "norm", "T": 16384, "H": 5120},
        # attention block (projections, rotary embedding, attention over packed documents) of the 0.5B model
        {"name": "attn_block_docs_0.5b", "kind": "attn_block", "arch": "qwen2.5-0.5b", "lens": DOCS_8K},
        # attention alone on long sequences, head size 128, 28 / 4 heads: long-context fine-tuning of a 7B model
        {"name": "attn_long_7b", "kind": "attn", "hq": 28, "hk": 4, "d": 128, "lens": "4096,4096", "grad": True},
        # gated MLP block of the 0.5B model on a micro-batch of 8 x 1024 tokens
        {"name": "mlp_0.5b", "kind": "mlp", "arch": "qwen2.5-0.5b", "T": 8192, "gelu": False},
        # language-model head with the fused cross-entropy, full vocabulary, a micro-batch of 4 x 1024 tokens
        {"name": "head_ce_0.5b", "kind": "head", "T": 4096, "H": 896, "V": 151936, "smoothing": 0.0, "z": 0.0},
        # loss on fp32 logits that a program already holds (drop-in replacement of torch's cross-entropy)
        {"name": "logits_ce_fp32", "kind": "logits_ce", "T": 2047, "V": 151936, "fp32": True, "smoothing": 0.0, "z": 0.0},
        # frozen gate | up projection with rank-16 adapters, the largest projection of a LoRA step
        {"name": "lora_gate_up_0.5b", "kind": "lora", "arch": "qwen2.5-0.5b", "proj": "gate_up", "T": 8192, "rank": 16},
        # token embedding, forward and backward; token frequencies follow Zipf's law, as in text
        {"name": "embed_0.5b", "kind": "embed", "T": 8192, "H": 896, "V": 151936},
        # optimizer step with global-norm clipping over two layers, the embedding and the final norm
        {"name": "adamw_0.5b", "kind": "adamw", "arch": "qwen2.5-0.5b", "layers": 2, "vocab": 151936, "fp32": False, "master": False},
        # MXFP8 gate | up projection of the 7B model: quantisation of both operands and the three GEMMs
        {"name": "mxfp8_gate_up_7b", "kind": "mxfp8", "arch": "qwen2.5-7b", "proj": "gate_up", "T": 4096},
    ]


# ------------------------------------------------------------------------------------------------ drawn cases
def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _lens(rng, total, most=64):
    """Document lengths that add up to `total`: equal rows, or log-normal lengths with a cut-off last one."""
    if rng.random() < 0.3:
        n = rng.choice([1, 2, 4, 8])
        return ",".join([str(max(1, total // n))] * n)
    mid, out = _log(rng, 32, 2048), []
    while sum(out) < total and len(out) < most:
        out.append(min(max(1, int(mid * math.exp(rng.gauss(0.0, 0.8)))), total - sum(out)))
    return ",".join(str(x) for x in out)


def _draw_one(rng):
    kind = rng.choice(["model", "norm", "attn_block", "attn", "mlp", "head", "logits_ce", "lora", "embed", "adamw", "mxfp8"])
    arch = rng.choice(PRESETS)
    if kind == "model":
        train = rng.random() < 0.6
        return {"kind": kind, "arch": rng.choice(["tiny-qwen2", "qwen2.5-0.5b", "llama-1b"]), "layers": rng.choice([1, 2, 4]),
                "vocab": rng.choice([4096, 32000]), "lens": _lens(rng, _log(rng, 48, 4096)), "train": train}
    if kind == "norm":
        return {"kind": kind, "T": _log(rng, 32, 32768), "H": rng.choice([256, 896, 1536, 2048, 3584, 5120, 8 * rng.randint(8, 1024)])}
    if kind == "attn_block":
        return {"kind": kind, "arch": arch, "lens": _lens(rng, _log(rng, 128, 8192))}
    if kind == "attn":
        hq, hk, d = rng.choice([(14, 2, 64), (12, 2, 128), (32, 8, 64), (24, 24, 64), (28, 4, 128), (40, 8, 128), (4, 2, 64)])
        return {"kind": kind, "hq": hq, "hk": hk, "d": d, "lens": _lens(rng, _log(rng, 128, 16384)), "grad": rng.random() < 0.7}
    if kind == "mlp":
        return {"kind": kind, "arch": arch, "T": _log(rng, 64, 16384), "gelu": rng.random() < 0.25}
    if kind == "head":
        return {"kind": kind, "T": _log(rng, 64, 4096), "H": rng.choice([256, 896, 1536, 2048]), "V": rng.choice([32000, 102400, 128256, 151936]),
                "smoothing": rng.choice([0.0, 0.0, 0.1]), "z": rng.choice([0.0, 0.0, 1e-4])}
    if kind == "logits_ce":
        return {"kind": kind, "T": _log(rng, 16, 8192), "V": rng.choice([32000, 102400, 128256, 151936, rng.randint(4000, 152000)]),
                "fp32": rng.random() < 0.5, "smoothing": rng.choice([0.0, 0.0, 0.1]), "z": rng.choice([0.0, 0.0, 1e-4])}
    if kind == "lora":
        return {"kind": kind, "arch": arch, "proj": rng.choice(["qkv", "o", "gate_up", "down"]), "T": _log(rng, 64, 8192),
                "rank": rng.choice([8, 16, 32, 64])}
    if kind == "embed":
        return {"kind": kind, "T": _log(rng, 32, 32768), "H": rng.choice([256, 896, 1536, 2048, 3584]), "V": rng.choice([32000, 102400, 128256, 151936])}
    if kind == "adamw":
        return {"kind": kind, "arch": rng.choice(["tiny-qwen2", "qwen2.5-0.5b", "qwen2.5-1.5b", "llama-1b"]), "layers": rng.choice([1, 2]),
                "vocab": rng.choice([0, 32000, 151936]), "fp32": rng.random() < 0.3, "master": rng.random() < 0.3}
    return {"kind": kind, "arch": arch, "proj": rng.choice(["qkv", "o", "gate_up", "down"]), "T": rng.choice([32, 1]) * _log(rng, 16, 256)}


def _cost(case):
    w = work(case)
    return max(w["flops"] / 1.0e15, w["bytes"] / 5e12)


def draw(rng):
    most = max(_cost(c) for c in listed())
    while True:
        c = _draw_one(rng)
        if _cost(c) <= most:
            return c


# ------------------------------------------------------------------------------------------------ inputs
class _Rand:
    def __init__(self, seed):
        self.g = torch.Generator(device=DEV).manual_seed(int(seed) * 7919 + 17)

    def normal(self, *shape, scale=1.0, dtype=BF):
        return torch.randn(*shape, device=DEV, generator=self.g).mul_(scale).to(dtype)

    def uniform(self, *shape):
        return torch.rand(*shape, device=DEV, generator=self.g)

    def tokens(self, n, vocab):
        """Token ids with frequency proportional to 1 / rank."""
        return (torch.exp(self.uniform(n) * math.log(vocab + 1)) - 1).long().clamp_(0, vocab - 1)

    def labels(self, n, vocab):
        """Targets, a fifth of them masked out as prompt tokens are."""
        y = self.tokens(n, vocab)
        return torch.where(self.uniform(n) < 0.2, torch.full_like(y, IGNORE), y)


def _config(case):
    cfg = ChronicalsConfig.from_model_name(case["arch"])
    over = {"hidden_act": "gelu_pytorch_tanh"} if case.get("gelu") else {}
    if case["kind"] == "model":
        over.update(num_hidden_layers=case["layers"], vocab_size=case["vocab"])
    return dataclasses.replace(cfg, **over)


def _doc_list(case):
    return [int(x) for x in case["lens"].split(",")]


def _documents(case):
    lens = _doc_list(case)
    bounds = [0]
    for n in lens:
        bounds.append(bounds[-1] + n)
    cu = torch.tensor(bounds, dtype=torch.int32, device=DEV)
    pos = torch.cat([torch.arange(n, device=DEV) for n in lens])
    return lens, cu, pos


def _proj(case):
    """(in features, {split: out features}, bias) of one fused projection of the architecture."""
    cfg = ChronicalsConfig.from_model_name(case["arch"])
    H, I, q, kv = cfg.hidden_size, cfg.intermediate_size, cfg.num_attention_heads * cfg.head_dim, cfg.num_key_value_heads * cfg.head_dim
    return {"qkv": (H, {"q_proj": q, "k_proj": kv, "v_proj": kv}, cfg.attention_bias), "o": (q, {"o_proj": H}, False),
            "gate_up": (H, {"gate_proj": I, "up_proj": I}, False), "down": (I, {"down_proj": H}, False)}[case["proj"]]


def _fill(module, r):
    """Weights of the scale that trained projections have: variance-preserving, norms near one, small biases."""
    with torch.no_grad():
        for name, p in module.named_parameters():
            if "embed" in name:
                p.copy_(r.normal(*p.shape, scale=0.02))
            elif name.endswith("norm.weight"):
                p.copy_(1 + r.normal(*p.shape, scale=0.1, dtype=torch.float32))
            elif p.dim() == 2:
                p.copy_(r.normal(*p.shape, scale=(0.02 if "lora_B" in name else p.shape[1] ** -0.5)))
            else:
                p.copy_(r.normal(*p.shape, scale=0.02))


def _adamw_shapes(case):
    cfg = ChronicalsConfig.from_model_name(case["arch"])
    H, I, q, kv = cfg.hidden_size, cfg.intermediate_size, cfg.num_attention_heads * cfg.head_dim, cfg.num_key_value_heads * cfg.head_dim
    layer = [(q + 2 * kv, H), (q + 2 * kv,), (H, q), (2 * I, H), (H, I), (H,), (H,)]
    return layer * case["layers"] + ([(case["vocab"], H)] if case["vocab"] else []) + [(H,)]


def _inputs(case, seed):
    """Everything `prepare` and `exact` start from; made from the seed alone."""
    r, k = _Rand(seed), case["kind"]
    s = {}
    if k == "model":
        lens, s["cu"], s["pos"] = _documents(case)
        T = sum(lens)
        s["model"] = CausalLM(_config(case), dtype=BF, device=DEV)
        _fill(s["model"], r)
        s["ids"], s["labels"] = r.tokens(T, case["vocab"]), r.labels(T, case["vocab"])
        s["lens"] = lens
    elif k == "norm":
        T, H = case["T"], case["H"]
        s.update(x=r.normal(T, H), w=(1 + r.normal(H, scale=0.1, dtype=torch.float32)).to(BF), dy=r.normal(T, H, scale=0.01),
                 dres=r.normal(T, H, scale=0.01))
    elif k == "attn_block":
        cfg = _config(case)
        s["lens"], s["cu"], s["pos"] = _documents(case)
        T = sum(s["lens"])
        s["block"] = Attention(cfg, BF, DEV)
        _fill(s["block"], r)
        s["cos"], s["sin"] = (t.contiguous() for t in ref.rope_cache(max(s["lens"]), cfg.head_dim, cfg.rope_theta, None, DEV))
        s.update(x=r.normal(T, cfg.hidden_size), res=r.normal(T, cfg.hidden_size), dy=r.normal(T, cfg.hidden_size, scale=0.01))
    elif k == "attn":
        s["lens"], s["cu"], _ = _documents(case)
        T, hq, hk, d = sum(s["lens"]), case["hq"], case["hk"], case["d"]
        s.update(x=r.normal(T, (hq + 2 * hk) * d), dy=r.normal(T, hq * d, scale=0.01))
    elif k == "mlp":
        cfg, T = _config(case), case["T"]
        s["block"] = MLP(cfg, BF, DEV)
        _fill(s["block"], r)
        s.update(x=r.normal(T, cfg.hidden_size), res=r.normal(T, cfg.hidden_size), dy=r.normal(T, cfg.hidden_size, scale=0.01))
    elif k == "head":
        s.update(x=r.normal(case["T"], case["H"]), w=r.normal(case["V"], case["H"], scale=0.02), labels=r.labels(case["T"], case["V"]))
    elif k == "logits_ce":
        s.update(x=r.normal(case["T"], case["V"], scale=2.0, dtype=torch.float32 if case["fp32"] else BF), labels=r.labels(case["T"], case["V"]))
    elif k in ("lora", "mxfp8"):
        n_in, splits, bias = _proj(case)
        fl = FusedLinear(n_in, splits, bias, BF, DEV)
        if k == "lora":
            for name in splits:
                fl.add_lora(name, case["rank"], 2.0 * case["rank"])
            fl.weight.requires_grad_(False)
            if fl.bias is not None:
                fl.bias.requires_grad_(False)
        _fill(fl, r)
        s["block"] = convert_model_to_fp8(fl, exclude_patterns=[]) if k == "mxfp8" else fl
        s.update(x=r.normal(case["T"], n_in), dy=r.normal(case["T"], sum(splits.values()), scale=0.01))
    elif k == "embed":
        s.update(ids=r.tokens(case["T"], case["V"]), w=r.normal(case["V"], case["H"], scale=0.02), dy=r.normal(case["T"], case["H"], scale=0.01))
    elif k == "adamw":
        dt = torch.float32 if case["fp32"] else BF
        s["params"] = [r.normal(*sh, scale=0.02, dtype=dt) for sh in _adamw_shapes(case)]
        s["grads"] = [r.normal(*sh, scale=1e-3, dtype=dt) for sh in _adamw_shapes(case)]
        s["m"] = [r.normal(*sh, scale=3e-4, dtype=torch.float32) for sh in _adamw_shapes(case)]
        s["v"] = [r.normal(*sh, scale=1e-3, dtype=torch.float32).square_() for sh in _adamw_shapes(case)]
    return s


ADAMW = dict(lr=1e-4, betas=(0.9, 0.95), eps=1e-8, weight_decay=0.01, max_grad_norm=1.0)
ADAMW_STEPS_DONE = 100


def prepare(case, seed):
    s = _inputs(case, seed)
    s["case"] = dict(case)
    k = case["kind"]
    if k == "model":
        s["model"].train(case["train"])
        s["model"].prepare_rope(max(s["lens"]), torch.device(DEV, torch.cuda.current_device()))
    elif k in ("norm", "head", "embed"):
        s["w"].requires_grad_()
    if "x" in s and case.get("grad", True):
        s["x"].requires_grad_()
    if k == "adamw":
        s["params"] = [torch.nn.Parameter(p) for p in s["params"]]
        opt = s["opt"] = FusedAdamW(s["params"], master_weights=case["master"], **ADAMW)
        opt.ensure_state()
        opt.step_count = ADAMW_STEPS_DONE
        for p, g, m, v in zip(s["params"], s.pop("grads"), s.pop("m"), s.pop("v")):
            p.grad = g
            opt.state[p]["exp_avg"].copy_(m)
            opt.state[p]["exp_avg_sq"].copy_(v)
    return s


# ------------------------------------------------------------------------------------------------ one pass
def _taken(tensors):
    """The gradients that the pass left, handed on as an optimizer would take them."""
    out = []
    for t in tensors:
        out.append(t.grad)
        t.grad = None
    return out


def run(s):
    case = s["case"]
    k = case["kind"]
    if k == "model":
        args = dict(position_ids=s["pos"], cu_seqlens=s["cu"], max_seqlen=max(s["lens"]), seqlens_host=s["lens"])
        if not case["train"]:
            with torch.no_grad():
                return {"logits": s["model"](s["ids"], **args).logits}
        o = s["model"](s["ids"], labels=s["labels"], return_logits=True, **args)
        o.loss.backward()
        return {"loss": o.loss.detach(), "logits": o.logits.detach(), "grads": _taken(list(s["model"].parameters()))}
    if k == "norm":
        y, r = ops.rmsnorm_residual(s["x"], s["w"])
        torch.autograd.backward((y, r), (s["dy"], s["dres"]))
        return {"y": y.detach(), "grads": _taken((s["x"], s["w"]))}
    if k == "attn_block":
        y = s["block"](s["x"], s["res"], s["cos"], s["sin"], s["pos"], s["cu"], max(s["lens"]), s["lens"])
        y.backward(s["dy"])
        return {"y": y.detach(), "grads": _taken([s["x"], *s["block"].parameters()])}
    if k == "attn":
        if not case["grad"]:
            with torch.no_grad():
                return {"y": ops.attention_qkv_packed(s["x"], s["cu"], case["hq"], case["hk"], case["d"], max(s["lens"]), s["lens"])}
        y = ops.attention_qkv_packed(s["x"], s["cu"], case["hq"], case["hk"], case["d"], max(s["lens"]), s["lens"])
        y.backward(s["dy"])
        return {"y": y.detach(), "grads": _taken((s["x"],))}
    if k == "mlp":
        y = s["block"](s["x"], s["res"])
        y.backward(s["dy"])
        return {"y": y.detach(), "grads": _taken([s["x"], *s["block"].parameters()])}
    if k == "head":
        loss = ops.linear_cross_entropy(s["x"], s["w"], s["labels"], None, IGNORE, case["smoothing"], case["z"])
        loss.backward()
        return {"loss": loss.detach(), "grads": _taken((s["x"], s["w"]))}
    if k == "logits_ce":
        loss = ops.cross_entropy_logits(s["x"], s["labels"], IGNORE, case["smoothing"], case["z"])
        loss.backward()
        return {"loss": loss.detach(), "grads": _taken((s["x"],))}
    if k in ("lora", "mxfp8"):
        y = s["block"](s["x"])
        y.backward(s["dy"])
        return {"y": y.detach(), "grads": _taken([s["x"], *(p for p in s["block"].parameters() if p.requires_grad)])}
    if k == "embed":
        y = ops.embedding(s["ids"], s["w"])
        y.backward(s["dy"])
        return {"y": y.detach(), "grads": _taken((s["w"],))}
    s["opt"].step()
    st = s["opt"].state
    return {"params": [p.detach() for p in s["params"]], "m": [st[p]["exp_avg"] for p in s["params"]],
            "v": [st[p]["exp_avg_sq"] for p in s["params"]]}


# ------------------------------------------------------------------------------------------------ what a pass needs
def _attn_flops(lens, hq, d, grad):
    return sum(2.0 * n * (n + 1) for n in lens) * hq * d * (3.5 if grad else 1.0)     # two products over the causal half, five more backward


def work(case):
    """Inputs read once, outputs written once (bf16 unless said otherwise); multiply-adds counted as two."""
    k = case["kind"]
    if k == "norm":
        T, H = case["T"], case["H"]
        return {"bytes": 10.0 * T * H, "flops": 12.0 * T * H}          # x, dy, dres in; y, dx out
    if k in ("attn_block", "attn", "model"):
        lens = _doc_list(case)
        T = sum(lens)
    if k == "attn":
        hq, hk, d, g = case["hq"], case["hk"], case["d"], case["grad"]
        io = T * ((hq + 2 * hk) * d * (2 if g else 1) + hq * d * (2 if g else 1))
        return {"bytes": 2.0 * io, "flops": _attn_flops(lens, hq, d, g)}
    if k == "attn_block":
        cfg = _config(case)
        hq, hk, d, H = cfg.num_attention_heads, cfg.num_key_value_heads, cfg.head_dim, cfg.hidden_size
        n = H * (hq + 2 * hk) * d + H * hq * d
        return {"bytes": 2.0 * (5 * T * H + 2 * n), "flops": 6.0 * T * n + _attn_flops(lens, hq, d, True)}
    if k == "model":
        cfg, train = _config(case), case["train"]
        hq, hk, d, H = cfg.num_attention_heads, cfg.num_key_value_heads, cfg.head_dim, cfg.hidden_size
        n = case["layers"] * (H * (hq + 2 * hk) * d + H * hq * d + 3 * H * cfg.intermediate_size) + H * case["vocab"]
        fl = (6.0 if train else 2.0) * T * n + case["layers"] * _attn_flops(lens, hq, d, train)
        return {"bytes": 2.0 * (n * (2 if train else 1) + T * case["vocab"]), "flops": fl}
    if k == "mlp":
        cfg, T = _config(case), case["T"]
        n = 3 * cfg.hidden_size * cfg.intermediate_size
        return {"bytes": 2.0 * (5 * T * cfg.hidden_size + 2 * n), "flops": 6.0 * T * n}
    if k == "head":
        T, H, V = case["T"], case["H"], case["V"]
        return {"bytes": 4.0 * (T * H + V * H), "flops": 6.0 * T * H * V}
    if k == "logits_ce":
        return {"bytes": (8.0 if case["fp32"] else 4.0) * case["T"] * case["V"], "flops": 8.0 * case["T"] * case["V"]}
    if k == "lora":
        n_in, splits, _ = _proj(case)
        T, n, R = case["T"], sum(splits.values()), case["rank"] * len(splits)
        a = R * n_in + case["rank"] * n
        return {"bytes": 2.0 * (T * 2 * (n_in + n) + n_in * n + 2 * a), "flops": 4.0 * T * n_in * n + 6.0 * T * a}
    if k == "mxfp8":
        n_in, splits, _ = _proj(case)
        T, n = case["T"], sum(splits.values())
        return {"bytes": 4.0 * (T * (n_in + n) + n_in * n), "flops": 6.0 * T * n_in * n}
    if k == "embed":
        T, H, V = case["T"], case["H"], case["V"]
        return {"bytes": 2.0 * (3 * T * H + V * H), "flops": 1.0 * T * H}
    n = sum(math.prod(sh) for sh in _adamw_shapes(case))
    per = (3 * (4 if case["fp32"] else 2)) + 16 + (8 if case["master"] and not case["fp32"] else 0)
    return {"bytes": float(per) * n, "flops": 15.0 * n}


def tolerance(case):
    """About four times what two correct implementations at bf16 inputs and outputs, fp32 accumulation, differ by."""
    k = case["kind"]
    if k == "model":
        return {"rel": 3e-2}                       # rounding of one layer travels through the others
    if k == "adamw":
        return {"rel": 1e-5 if case["fp32"] else 1e-3}
    if k == "logits_ce":
        return {"rel": 1e-5 if case["fp32"] else 5e-3}
    return {"rel": 1e-2}


# ------------------------------------------------------------------------------------------------ the same in 64 bits
D = torch.float64


def _leaf(t):
    return t.detach().to(D).requires_grad_()


def _rms64(x, w, eps=1e-6):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps) * w


def _rope64(x, cos, sin):
    a, b = x.chunk(2, dim=-1)
    c, s = cos[:, None, :], sin[:, None, :]
    return torch.cat((a * c - b * s, b * c + a * s), dim=-1)


def _attend64(q, k, v, lens):
    """Causal attention per document and key head; q [T, hq, d], k and v [T, hk, d]."""
    hq, hk, d = q.shape[1], k.shape[1], q.shape[2]
    docs, at = [], 0
    for n in lens:
        heads = []
        mask = torch.ones(n, n, dtype=torch.bool, device=q.device).triu_(1)
        for h in range(hk):
            qq = q[at:at + n, h * (hq // hk):(h + 1) * (hq // hk)].transpose(0, 1)
            p = torch.softmax((qq @ k[at:at + n, h].t() * d ** -0.5).masked_fill(mask, -math.inf), dim=-1)
            heads.append((p @ v[at:at + n, h]).transpose(0, 1))
        docs.append(torch.cat(heads, dim=1))
        at += n
    return torch.cat(docs, dim=0)


def _attn_block64(cfg, x, res, p, cos, sin, pos, lens, name=""):
    hq, hk, d = cfg.num_attention_heads, cfg.num_key_value_heads, cfg.head_dim
    qkv = x @ p[name + "qkv_proj.weight"].t()
    if name + "qkv_proj.bias" in p:
        qkv = qkv + p[name + "qkv_proj.bias"]
    q, k, v = (t.reshape(x.shape[0], -1, d) for t in qkv.split([hq * d, hk * d, hk * d], dim=1))
    c, s = cos.to(D)[pos], sin.to(D)[pos]
    o = _attend64(_rope64(q, c, s), _rope64(k, c, s), v, lens)
    return o.reshape(x.shape[0], hq * d) @ p[name + "o_proj.weight"].t() + res


def _mlp64(x, res, p, gelu, name=""):
    g, u = (x @ p[name + "gate_up_proj.weight"].t()).chunk(2, dim=1)
    a = torch.nn.functional.gelu(g, approximate="tanh") if gelu else torch.nn.functional.silu(g)
    return (a * u) @ p[name + "down_proj.weight"].t() + res


def _ce64(logits, y, smoothing, z):
    """Sum over the valid rows of the smoothed cross-entropy with z-loss, over their number."""
    ok = y != IGNORE
    lse = torch.logsumexp(logits, dim=-1)
    row = lse - logits.gather(1, y.clamp_min(0)[:, None])[:, 0]
    if smoothing:
        row = (1 - smoothing) * row + smoothing * (lse - logits.mean(dim=-1))
    return torch.where(ok, row + z * lse.square(), torch.zeros_like(row)).sum() / ok.sum().clamp_min(1)


def _mx64(x, fmt):
    """x rounded to 8-bit floats with one power-of-two scale for each 32 values of the last dimension."""
    top, dt = (448.0, torch.float8_e4m3fn) if fmt == "e4m3" else (57344.0, torch.float8_e5m2)
    n = x.shape[-1]
    b = torch.nn.functional.pad(x.float(), (0, -n % 32)).unflatten(-1, (-1, 32))
    m, e = torch.frexp(b.abs().amax(-1, keepdim=True) / top)
    e = torch.where(m == 0.5, e - 1, e).to(D)
    q = (b.to(D) * torch.exp2(-e)).float().to(dt).to(D) * torch.exp2(e)
    return q.flatten(-2)[..., :n]


def exact(case, seed):
    if work(case)["flops"] > 4e13:
        return None
    s, k = _inputs(case, seed), case["kind"]
    if k == "adamw":
        b1, b2 = ADAMW["betas"]
        t = ADAMW_STEPS_DONE + 1
        norm = sum(g.to(D).square().sum() for g in s["grads"]).sqrt()
        clip = (ADAMW["max_grad_norm"] / (norm + 1e-6)).clamp(max=1.0)
        out = {"params": [], "m": [], "v": []}
        for p, g, m, v in zip(s["params"], s["grads"], s["m"], s["v"]):
            g = g.to(D) * clip
            m, v = b1 * m.to(D) + (1 - b1) * g, b2 * v.to(D) + (1 - b2) * g * g
            p = p.to(D) * (1 - ADAMW["lr"] * ADAMW["weight_decay"])
            out["params"].append(p - ADAMW["lr"] * (m / (1 - b1 ** t)) / ((v / (1 - b2 ** t)).sqrt() + ADAMW["eps"]))
            out["m"].append(m)
            out["v"].append(v)
        return out
    if k == "embed":
        dw = torch.zeros(case["V"], case["H"], dtype=D, device=DEV).index_add_(0, s["ids"], s["dy"].to(D))
        return {"y": s["w"].to(D)[s["ids"]], "grads": [dw]}
    if k == "mxfp8":
        fl, x, dy = s["block"], s["x"], s["dy"]
        w = fl.weight.detach()
        y = _mx64(x, "e4m3") @ _mx64(w, "e4m3").t()
        g = [_mx64(dy, "e5m2") @ _mx64(w.t(), "e4m3").t(), _mx64(dy.t(), "e5m2") @ _mx64(x.t(), "e4m3").t()]
        if fl.bias is not None:
            y = y + fl.bias.detach().to(D)
            g.append(dy.to(D).sum(0))
        return {"y": y, "grads": g}
    if k == "model":
        m, cfg = s["model"], _config(case)
        p = {n: _leaf(t) for n, t in m.named_parameters()}
        cos, sin = ref.rope_cache(max(s["lens"]), cfg.head_dim, cfg.rope_theta, cfg.rope_scaling, DEV)
        h = p["model.embed_tokens.weight"][s["ids"]]
        for i in range(case["layers"]):
            n = "model.layers.%d." % i
            h = _attn_block64(cfg, _rms64(h, p[n + "input_layernorm.weight"], cfg.rms_norm_eps), h, p, cos, sin, s["pos"], s["lens"], n + "self_attn.")
            h = _mlp64(_rms64(h, p[n + "post_attention_layernorm.weight"], cfg.rms_norm_eps), h, p, False, n + "mlp.")
        logits = _rms64(h, p["model.norm.weight"], cfg.rms_norm_eps) @ p["model.embed_tokens.weight"].t()
        logits = logits.view(1, len(s["ids"]), -1)
        if not case["train"]:
            return {"logits": logits.detach()}
        y = torch.cat((s["labels"][1:], s["labels"].new_full((1,), IGNORE)))
        loss = _ce64(logits[0], y, 0.0, 0.0)
        loss.backward()
        return {"loss": loss.detach(), "logits": logits.detach(), "grads": [p[n].grad for n, _ in m.named_parameters()]}
    x = _leaf(s["x"])
    if k == "norm":
        w = _leaf(s["w"])
        y = _rms64(x, w)
        torch.autograd.backward((y, x * 1.0), (s["dy"].to(D), s["dres"].to(D)))
        return {"y": y.detach(), "grads": [x.grad, w.grad]}
    if k == "attn":
        hq, hk, d = case["hq"], case["hk"], case["d"]
        q, kk, v = (t.reshape(x.shape[0], -1, d) for t in x.split([hq * d, hk * d, hk * d], dim=1))
        y = _attend64(q, kk, v, s["lens"]).reshape(x.shape[0], hq * d)
        if not case["grad"]:
            return {"y": y.detach()}
        y.backward(s["dy"].to(D))
        return {"y": y.detach(), "grads": [x.grad]}
    if k == "head":
        w = _leaf(s["w"])
        loss = _ce64(x @ w.t(), s["labels"], case["smoothing"], case["z"])
        loss.backward()
        return {"loss": loss.detach(), "grads": [x.grad, w.grad]}
    if k == "logits_ce":
        loss = _ce64(x, s["labels"], case["smoothing"], case["z"])
        loss.backward()
        return {"loss": loss.detach(), "grads": [x.grad]}
    p = {n: _leaf(t) for n, t in s["block"].named_parameters()}
    if k == "attn_block":
        y = _attn_block64(_config(case), x, s["res"].to(D), p, s["cos"], s["sin"], s["pos"], s["lens"])
    elif k == "mlp":
        y = _mlp64(x, s["res"].to(D), p, case["gelu"])
    else:
        fl = s["block"]
        y = x @ p["weight"].t()
        if "bias" in p:
            y = y + p["bias"]
        y = y + torch.cat([fl.lora_scaling[n] * (x @ p["lora_A." + n].t()) @ p["lora_B." + n].t() for n in fl.splits], dim=1)
    y.backward(s["dy"].to(D))
    return {"y": y.detach(), "grads": [x.grad, *(p[n].grad for n, t in s["block"].named_parameters() if t.requires_grad)]}
