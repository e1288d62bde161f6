"""The work that a program built on this framework gives it, as cases that can be timed and checked.

Kinds (every one through an entry point that the models, the loader or a user's own module calls):

* ``linear``     ``LowBitLinear.forward``: one projection of a decoder layer, from one row (decoding) over small batches to prompts;
* ``mlp``        ``mlp_silu_forward``: gate, up, activation, down of a decoder layer;
* ``experts``    ``LowBitExperts.forward``: the routed feed-forwards of a mixture-of-experts layer;
* ``train``      ``MatMulLowBit`` forward and backward: an adapter's training step through a frozen low-bit projection;
* ``attention``  ``scaled_dot_product_attention`` over the 8-bit key/value cache: one new token per sequence, or a whole prompt;
* ``recurrence`` ``gated_delta_rule``: the linear-attention half of the framework's hybrid layers;
* ``step``       the recorded decode step behind ``generate()``, whole model, logits out.

Sizes are those of the Llama-2-7B / Mistral-7B / Mixtral layers that the tests and the benchmark use, or generic ones of that range.
"""
import math

import torch

QTYPES = ("sym_int4", "asym_int4", "nf4", "fp8_e4m3", "fp8_e5m2", "fp6")
BLOCK_BYTES = {"sym_int4": 34, "asym_int4": 36, "nf4": 34, "fp8_e4m3": 66, "fp8_e5m2": 66, "fp6": 50}
DTYPES = {"fp16": torch.float16, "bf16": torch.bfloat16, "fp32": torch.float32}
DEVICE = "cuda"


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # the smallest call of a decode step: an output projection at batch 1, where the launch is most of the time
        {"name": "token_linear", "kind": "linear", "rows": 1, "n": 4096, "k": 4096, "qtype": "sym_int4", "dtype": "fp16"},
        # sixteen sequences decoded together, 8-bit weights, the merged q/k/v projection of a grouped-query layer
        {"name": "batch_linear_fp8", "kind": "linear", "rows": 16, "n": 6144, "k": 4096, "qtype": "fp8_e4m3", "dtype": "bf16"},
        # a serving batch that is no power of two, 4-bit weights with minima
        {"name": "batch_linear_40", "kind": "linear", "rows": 40, "n": 11008, "k": 4096, "qtype": "asym_int4", "dtype": "fp16"},
        # the headline benchmark's prompt of 512 tokens through the down projection
        {"name": "prompt_linear", "kind": "linear", "rows": 512, "n": 4096, "k": 11008, "qtype": "sym_int4", "dtype": "fp16"},
        # a 32-bit model's prompt with the 32-bit contract of the reference's matmul (no cast to half precision)
        {"name": "prompt_linear_fp32", "kind": "linear", "rows": 200, "n": 4096, "k": 4096, "qtype": "sym_int4", "dtype": "fp32"},
        # a long prompt of ragged length through a whole feed-forward: the largest case
        {"name": "long_mlp", "kind": "mlp", "rows": 4000, "hidden": 4096, "inter": 14336, "qtype": "sym_int4", "dtype": "bf16"},
        # a prompt through a mixture of experts
        {"name": "prompt_experts", "kind": "experts", "rows": 512, "hidden": 4096, "inter": 14336, "experts": 8, "top_k": 2, "qtype": "sym_int4",
         "dtype": "bf16"},
        # a training step of an adapter on a frozen 4-bit normal-float projection
        {"name": "train_linear", "kind": "train", "rows": 1024, "n": 11008, "k": 4096, "qtype": "nf4", "dtype": "bf16"},
        # eight sequences at 4000 held tokens, one new token each
        {"name": "token_attention", "kind": "attention", "batch": 8, "heads": 32, "kv_heads": 8, "new": 1, "held": 4000, "dim": 128, "dtype": "fp16"},
        # a prompt of 4000 tokens, causal
        {"name": "prompt_attention", "kind": "attention", "batch": 1, "heads": 32, "kv_heads": 8, "new": 4000, "held": 0, "dim": 128, "dtype": "bf16"},
        # a prompt through a hybrid layer's delta rule
        {"name": "prompt_recurrence", "kind": "recurrence", "batch": 1, "new": 2048, "heads": 16, "kv_heads": 4, "dim": 128, "vdim": 128, "dtype": "bf16"},
        # one decoded token of a model with the headline benchmark's layers (eight of them) behind a prompt of 512 tokens
        {"name": "token_step", "kind": "step", "batch": 1, "prompt": 512, "layers": 8, "hidden": 4096, "inter": 11008, "heads": 32, "kv_heads": 32,
         "vocab": 32000, "qtype": "sym_int4", "dtype": "fp16"},
    ]


def _log(rng, lo, hi, unit=1):
    """a whole number spread evenly over the logarithm of [lo, hi], in units"""
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))) / unit)) * unit))


def _cost(case):
    w = work(case)
    return max(w["bytes"], w["flops"] / 200)


def draw(rng):
    most = max(_cost(c) for c in listed())
    while True:
        kind = rng.choice(("linear", "linear", "linear", "mlp", "experts", "train", "attention", "attention", "recurrence", "step"))
        half, any_q = rng.choice(("fp16", "bf16")), rng.choice(QTYPES)
        if kind == "linear":
            dtype = rng.choice(("fp16", "bf16", "fp16", "bf16", "fp32"))
            case = {"rows": _log(rng, 1, 4096 if dtype != "fp32" else 512), "n": _log(rng, 1024, 32000, 64), "k": _log(rng, 1024, 14336, 64), "qtype": any_q,
                    "dtype": dtype}
        elif kind == "mlp":
            case = {"rows": _log(rng, 1, 4096), "hidden": _log(rng, 1024, 8192, 128), "inter": _log(rng, 2048, 14336, 128), "qtype": any_q, "dtype": half}
        elif kind == "experts":
            case = {"rows": _log(rng, 1, 2048), "hidden": _log(rng, 1024, 4096, 128), "inter": _log(rng, 1024, 14336, 128), "experts": rng.choice((4, 8, 16)),
                    "top_k": rng.choice((1, 2, 4)), "qtype": rng.choice(("sym_int4", "asym_int4", "fp8_e4m3", "fp6")), "dtype": half}
        elif kind == "train":
            case = {"rows": _log(rng, 16, 4096), "n": _log(rng, 1024, 14336, 128), "k": _log(rng, 1024, 14336, 128), "qtype": any_q, "dtype": half}
        elif kind == "attention":
            kv = rng.choice((1, 4, 8, 32))
            case = {"batch": _log(rng, 1, 16), "heads": kv * rng.choice([g for g in (1, 2, 4, 8) if 4 <= kv * g <= 32]), "kv_heads": kv, "new": 1,
                    "held": _log(rng, 64, 16384), "dim": 128, "dtype": half}
            if rng.random() < 0.5:
                case.update(batch=rng.choice((1, 1, 2, 4)), new=_log(rng, 2, 6000), held=rng.choice((0, 0, 0, 777)))
        elif kind == "recurrence":
            kv = rng.choice((2, 4, 8))
            case = {"batch": rng.choice((1, 1, 2, 4)), "new": _log(rng, 16, 4096), "heads": kv * rng.choice((1, 2, 4)), "kv_heads": kv,
                    "dim": rng.choice((64, 128)), "vdim": rng.choice((64, 128, 256)), "dtype": rng.choice(("bf16", "bf16", "fp16", "fp32"))}
        else:
            kv = rng.choice((4, 8, 16))
            heads = kv * rng.choice((1, 2))
            case = {"batch": _log(rng, 1, 8), "prompt": _log(rng, 17, 1500), "layers": rng.choice((2, 4, 6)), "hidden": heads * 128,
                    "inter": _log(rng, 2048, 11008, 128), "heads": heads, "kv_heads": kv, "vocab": 32000, "qtype": any_q, "dtype": "fp16"}
        case = {"kind": kind, **case}
        if _cost(case) <= most:
            return case


# ------------------------------------------------------------------ inputs, from the seed alone
class _Draws:
    def __init__(self, seed):
        self.g = torch.Generator(device=DEVICE).manual_seed(seed)

    def normal(self, *shape, std=1.0, dtype=torch.float32):
        return torch.empty(*shape, dtype=torch.float32, device=DEVICE).normal_(0.0, std, generator=self.g).to(dtype)

    def ints(self, hi, *shape):
        return torch.randint(0, hi, shape, generator=self.g, device=DEVICE)


def _weight(d, n, k):
    return d.normal(n, k, std=0.02)


def _low_bit(w, qtype, half=True):
    from ipex_llm_b200.transformers.low_bit_linear import FP4Params, LowBitLinear, ggml_tensor_qtype
    n, k = w.shape
    with torch.device("meta"):
        lin = LowBitLinear(k, n, ggml_tensor_qtype[qtype], bias=False, conver_to_half=half)
    lin._parameters["weight"] = FP4Params(w, qtype=ggml_tensor_qtype[qtype]).to(DEVICE)
    return lin.eval()


def _routing(case, d):
    logits = d.normal(case["rows"], case["experts"])
    top = torch.topk(torch.softmax(logits, -1), case["top_k"], dim=-1)
    return top.indices, (top.values / top.values.sum(-1, keepdim=True))


class _Mlp(torch.nn.Module):
    def __init__(self, gate, up, down):
        super().__init__()
        self.gate_proj, self.up_proj, self.down_proj, self.act_fn = gate, up, down, torch.nn.SiLU()


class _FusedExperts(torch.nn.Module):
    """the layout a checkpoint's experts have before conversion"""

    def __init__(self, gate_up, down):
        super().__init__()
        self.gate_up_proj = torch.nn.Parameter(gate_up, requires_grad=False)
        self.down_proj = torch.nn.Parameter(down, requires_grad=False)
        self.act_fn = torch.nn.SiLU()


def _attention_inputs(case, seed):
    d = _Draws(seed)
    B, L, D, dt = case["batch"], case["held"] + case["new"], case["dim"], DTYPES[case["dtype"]]
    # the query is the transposed view of the projection's output, as in the models; the cache holds e5m2 bytes
    q = d.normal(B, case["new"], case["heads"], D, dtype=dt).transpose(1, 2)
    k, v = (d.normal(B, case["kv_heads"], L, D).to(torch.float8_e5m2).view(torch.uint8) for _ in range(2))
    return q, k, v


def _recurrence_inputs(case, seed):
    d = _Draws(seed)
    B, S, G, H, D, V = (case[x] for x in ("batch", "new", "kv_heads", "heads", "dim", "vdim"))
    dt = DTYPES[case["dtype"]]
    conv = torch.nn.functional.silu(d.normal(B, S, 2 * G * D + H * V)).to(dt)      # what the short convolution hands over
    proj = d.normal(B, S, 2 * H, dtype=dt)                                           # the gates' logits
    a_log, bias = (d.normal(H, std=0.5) - 1.0).to(dt), d.normal(H, std=0.5, dtype=dt)
    return conv, proj, a_log, bias


def _step_model(case, d):
    import transformers
    from ipex_llm.transformers import AutoModelForCausalLM
    from ipex_llm_b200.optimize import low_memory_init
    dt = DTYPES[case["dtype"]]
    cfg = transformers.LlamaConfig(hidden_size=case["hidden"], intermediate_size=case["inter"], num_hidden_layers=case["layers"],
                                   num_attention_heads=case["heads"], num_key_value_heads=case["kv_heads"], vocab_size=case["vocab"],
                                   max_position_embeddings=4096, rms_norm_eps=1e-5, tie_word_embeddings=False)
    with low_memory_init():
        model = transformers.LlamaForCausalLM(cfg)
    for mod in model.modules():
        for name, p in list(mod._parameters.items()):
            if p is not None:
                mod._parameters[name] = torch.nn.Parameter(torch.ones(p.shape, dtype=dt, device=DEVICE) if p.dim() == 1
                                                           else d.normal(*p.shape, std=0.02, dtype=dt), requires_grad=False)
    model.model.rotary_emb = type(model.model.rotary_emb)(cfg).to(DEVICE)
    return AutoModelForCausalLM.from_model(model.eval(), low_bit=case["qtype"]).to(DEVICE)


def prepare(case, seed):
    kind = case["kind"]
    dt = DTYPES[case["dtype"]]
    d = _Draws(seed)
    if kind == "linear":
        lin = _low_bit(_weight(d, case["n"], case["k"]), case["qtype"], half=case["dtype"] != "fp32")
        return {"case": case, "lin": lin, "x": d.normal(1, case["rows"], case["k"], dtype=dt)}
    if kind == "mlp":
        H, I = case["hidden"], case["inter"]
        mlp = _Mlp(*(_low_bit(_weight(d, n, k), case["qtype"]) for n, k in ((I, H), (I, H), (H, I)))).eval()
        return {"case": case, "mlp": mlp, "x": d.normal(1, case["rows"], H, dtype=dt)}
    if kind == "experts":
        from ipex_llm_b200.transformers.low_bit_linear import ggml_tensor_qtype
        from ipex_llm_b200.transformers.models.mixtral import LowBitExperts
        E, H, I = case["experts"], case["hidden"], case["inter"]
        fused = _FusedExperts(d.normal(E, 2 * I, H, std=0.02, dtype=dt), d.normal(E, H, I, std=0.02, dtype=dt)).eval()
        experts = LowBitExperts.from_fused(fused, ggml_tensor_qtype[case["qtype"]])
        return {"case": case, "experts": experts, "x": d.normal(case["rows"], H, dtype=dt), "routing": _routing(case, d)}
    if kind == "train":
        lin = _low_bit(_weight(d, case["n"], case["k"]), case["qtype"])
        return {"case": case, "weight": lin.weight, "x": d.normal(1, case["rows"], case["k"], dtype=dt),
                "grad": d.normal(1, case["rows"], case["n"], dtype=dt)}
    if kind == "attention":
        q, k, v = _attention_inputs(case, seed)
        return {"case": case, "q": q, "k": k, "v": v}
    if kind == "recurrence":
        conv, proj, a_log, bias = _recurrence_inputs(case, seed)
        B, H = case["batch"], case["heads"]
        return {"case": case, "conv": conv, "proj": proj, "a_log": a_log, "bias": bias,
                "state": torch.zeros(B, H, case["dim"], case["vdim"], dtype=torch.float32, device=DEVICE),
                "pad": torch.zeros(B, dtype=torch.int32, device=DEVICE)}
    if kind == "step":
        from ipex_llm_b200.transformers.decode_graph import get_decode_graph
        model = _step_model(case, d)
        ids = d.ints(case["vocab"], case["batch"], case["prompt"])
        step = get_decode_graph(model, case["batch"], case["prompt"] + 32)
        with torch.no_grad():
            model(input_ids=ids, past_key_values=step.bind_cache(), use_cache=True)
        # the token that follows the prompt, as the program's own choice of it: one logit above the others
        chosen = torch.zeros(case["batch"], case["vocab"], dtype=dt, device=DEVICE)
        chosen.scatter_(1, d.ints(case["vocab"], case["batch"], 1), 1.0)
        return {"case": case, "model": model, "step": step, "chosen": chosen}
    raise ValueError(kind)


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "linear":
        with torch.no_grad():
            return state["lin"](state["x"])
    if kind == "mlp":
        from ipex_llm_b200.transformers.models.common import mlp_silu_forward
        with torch.no_grad():
            return mlp_silu_forward(state["mlp"], state["x"])
    if kind == "experts":
        with torch.no_grad():
            return state["experts"](state["x"], *state["routing"])
    if kind == "train":
        from ipex_llm_b200.transformers.low_bit_linear import MatMulLowBit
        x = state["x"].detach().requires_grad_(True)
        y = MatMulLowBit.apply(x, state["weight"], case["n"])
        (grad,) = torch.autograd.grad(y, x, state["grad"])
        return y.detach(), grad
    if kind == "attention":
        from ipex_llm_b200.transformers.kv import scaled_dot_product_attention
        with torch.no_grad():
            return scaled_dot_product_attention(state["q"], state["k"], state["v"], None, case["new"] > 1, case["dim"] ** -0.5)
    if kind == "recurrence":
        from ipex_llm_b200.transformers.models.mixer_ops import gated_delta_rule
        state["state"].zero_()                                                        # the sequence begins here
        o = gated_delta_rule(state["conv"], case["kv_heads"], case["heads"], case["dim"], case["vdim"], state["proj"], 0, case["heads"],
                             state["a_log"], state["bias"], state["state"], 0, state["pad"])
        return o, state["state"]
    step = state["step"]
    step.start(state["chosen"], case["prompt"])
    step.replay()
    return step.logits


# ------------------------------------------------------------------ what a pass cannot do without
def _packed(n, k, qtype):
    return n * (k // 64) * BLOCK_BYTES[qtype]


def work(case):
    kind = case["kind"]
    e = 4 if case["dtype"] == "fp32" else 2
    if kind == "linear":
        m, n, k = case["rows"], case["n"], case["k"]
        return {"bytes": _packed(n, k, case["qtype"]) + e * m * (n + k), "flops": 2 * m * n * k}
    if kind == "mlp":
        m, h, i = case["rows"], case["hidden"], case["inter"]
        return {"bytes": 2 * _packed(i, h, case["qtype"]) + _packed(h, i, case["qtype"]) + 2 * e * m * h, "flops": 6 * m * h * i}
    if kind == "experts":
        m, h, i, t = case["rows"], case["hidden"], case["inter"], case["top_k"]
        used = case["experts"] * (1 - (1 - t / case["experts"]) ** m)                 # experts that any row is routed to, on average
        one = 2 * _packed(i, h, case["qtype"]) + _packed(h, i, case["qtype"])
        return {"bytes": int(used * one) + 2 * e * m * h + 12 * m * t, "flops": 6 * m * t * h * i}
    if kind == "train":
        m, n, k = case["rows"], case["n"], case["k"]
        return {"bytes": 2 * _packed(n, k, case["qtype"]) + 2 * e * m * (n + k), "flops": 4 * m * n * k}
    if kind == "attention":
        b, s, p, h, g, d = (case[x] for x in ("batch", "new", "held", "heads", "kv_heads", "dim"))
        pairs = s * p + s * (s + 1) // 2
        return {"bytes": b * (2 * g * (s + p) * d + 2 * e * h * s * d), "flops": 4 * b * h * d * pairs}
    if kind == "recurrence":
        b, s, h, g, d, v = (case[x] for x in ("batch", "new", "heads", "kv_heads", "dim", "vdim"))
        return {"bytes": b * s * (e * (2 * g * d + h * v + 2 * h) + 4 * h * v) + 4 * b * h * d * v, "flops": 6 * b * s * h * d * v}
    b, p, h, i, L = (case[x] for x in ("batch", "prompt", "hidden", "inter", "layers"))
    kvw, q = case["kv_heads"] * 128, case["qtype"]
    weights = L * (_packed(h + 2 * kvw, h, q) + _packed(h, h, q) + 2 * _packed(i, h, q) + _packed(h, i, q)) + _packed(case["vocab"], h, q)
    count = L * (2 * h * h + 2 * kvw * h + 3 * h * i) + case["vocab"] * h
    return {"bytes": weights + b * L * 2 * kvw * p + b * e * case["vocab"], "flops": 2 * b * count + b * L * 4 * h * p}


def tolerance(case):
    kind, dtype = case["kind"], case["dtype"]
    # measured against exact(): about four times what is seen (single products 3e-4 / 2.4e-3 in fp16 / bf16, feed-forwards with
    # their two intermediates in 16 bits twice that)
    if kind == "recurrence":
        return {"rel": 2e-6}
    if kind == "step":
        # every layer rounds to 16 bits and the prompt's keys and values to e5m2: a change of one rounding in the prompt
        # moves a few of the cache's bytes by a whole step of that format (6e-3 seen between two ways to cut a prompt, fp16)
        return {"rel": 2.5e-2}
    if dtype == "fp32":
        return {"rel": 2e-6 if case["qtype"] != "nf4" else 1e-5}                      # nf4: its table is held as two bf16 planes
    if kind in ("mlp", "experts"):
        return {"rel": 2.6e-3 if dtype == "fp16" else 2e-2}
    return {"rel": 1.2e-3 if dtype == "fp16" else 1e-2}


# ------------------------------------------------------------------ the same in 64 bits, in plain torch
NF4 = (-1.0, -0.6961928009986877, -0.5250730514526367, -0.39491748809814453, -0.28444138169288635, -0.18477343022823334, -0.09105003625154495, 0.0,
       0.07958029955625534, 0.16093020141124725, 0.24611230194568634, 0.33791524171829224, 0.44070982933044434, 0.5626170039176941, 0.7229568362236023, 1.0)


def _mini(x, exp_bits, man_bits, bias, top):
    """round to nearest even in a small float format, saturating"""
    a = x.abs()
    e = torch.frexp(a)[1].to(torch.float32) - 1.0
    ulp = torch.exp2(torch.clamp(e, min=float(1 - bias)) - man_bits)
    return torch.copysign(torch.clamp(torch.round(a / ulp) * ulp, max=top), x)


def _stored(w, qtype):
    """float64 weights after a round trip through blocks of 64 of ``qtype``"""
    n, k = w.shape
    x = w.to(torch.float32).view(-1, 64)
    if qtype == "sym_int4":
        at = x.abs().argmax(1, keepdim=True)
        scale = x.gather(1, at) * -0.125
    elif qtype == "asym_int4":
        low = x.amin(1, keepdim=True)
        scale = torch.div(x.amax(1, keepdim=True) - low, torch.full_like(low, 15.0))      # a tensor: a number would become a reciprocal
    else:
        top = {"nf4": 1.0, "fp8_e4m3": 448.0, "fp8_e5m2": 57344.0, "fp6": 28.0}[qtype]
        scale = x.abs().amax(1, keepdim=True)
        scale = torch.div(scale, torch.full_like(scale, top))
    inverse = torch.where(scale != 0, 1.0 / scale, torch.zeros_like(scale))
    d = scale.half().double()
    if qtype == "sym_int4":
        code = torch.clamp(torch.floor(x * inverse + 8.5), max=15.0).double() - 8.0
        return (code * d).view(n, k)
    if qtype == "asym_int4":
        code = torch.clamp(torch.floor((x - low) * inverse + 0.5), max=15.0).double()
        return (code * d + low.half().double()).view(n, k)
    if qtype == "nf4":
        table = torch.tensor(NF4, dtype=torch.float32, device=w.device)
        code = torch.bucketize(x * inverse, (table[1:] + table[:-1]) * 0.5)
        return (table.double()[code] * d).view(n, k)
    fmt = {"fp8_e4m3": (4, 3, 7, 448.0), "fp8_e5m2": (5, 2, 15, 57344.0), "fp6": (3, 2, 3, 28.0)}[qtype]
    return (_mini(x * inverse, *fmt).double() * d).view(n, k)


def _exact_attention(case, seed):
    q, k, v = _attention_inputs(case, seed)
    B, H, S, D = q.shape
    k, v = (t.view(torch.float8_e5m2).double() for t in (k, v))
    out = torch.empty(B, H, S, D, dtype=torch.float64, device=DEVICE)
    causal = case["new"] > 1
    ahead = torch.ones(S, k.shape[2], dtype=torch.bool, device=DEVICE).triu(case["held"] + 1) if causal else None
    for b in range(B):
        for h in range(H):
            g = h // (H // case["kv_heads"])
            s = (q[b, h].double() @ k[b, g].T) * D ** -0.5
            if causal:
                s.masked_fill_(ahead, float("-inf"))
            out[b, h] = torch.softmax(s, -1) @ v[b, g]
    return out


def _exact_recurrence(case, seed):
    conv, proj, a_log, bias = _recurrence_inputs(case, seed)
    B, S, G, H, D, V = (case[x] for x in ("batch", "new", "kv_heads", "heads", "dim", "vdim"))
    c, p = conv.double(), proj.double()

    def unit(t):
        return t * torch.rsqrt((t * t).sum(-1, keepdim=True) + 1e-6)
    q = (unit(c[..., :G * D].view(B, S, G, D)) * D ** -0.5).repeat_interleave(H // G, 2)
    k = unit(c[..., G * D:2 * G * D].view(B, S, G, D)).repeat_interleave(H // G, 2)
    v = c[..., 2 * G * D:].view(B, S, H, V)
    beta = torch.sigmoid(p[..., :H])
    decay = torch.exp(-torch.exp(a_log.double()) * torch.nn.functional.softplus(p[..., H:] + bias.double()))
    M = torch.zeros(B, H, D, V, dtype=torch.float64, device=DEVICE)
    o = torch.empty(B, S, H, V, dtype=torch.float64, device=DEVICE)
    for t in range(S):
        M *= decay[:, t, :, None, None]
        u = beta[:, t, :, None] * (v[:, t] - torch.einsum("bhdv,bhd->bhv", M, k[:, t]))
        M += k[:, t, :, :, None] * u[:, :, None, :]
        o[:, t] = torch.einsum("bhdv,bhd->bhv", M, q[:, t])
    return o, M


def exact(case, seed):
    kind = case["kind"]
    d = _Draws(seed)
    dt = DTYPES[case["dtype"]]
    if kind == "linear":
        w = _stored(_weight(d, case["n"], case["k"]), case["qtype"])
        return d.normal(1, case["rows"], case["k"], dtype=dt).double() @ w.T
    if kind == "mlp":
        H, I = case["hidden"], case["inter"]
        gate, up, down = (_stored(_weight(d, n, k), case["qtype"]) for n, k in ((I, H), (I, H), (H, I)))
        x = d.normal(1, case["rows"], H, dtype=dt).double()
        return (torch.nn.functional.silu(x @ gate.T) * (x @ up.T)) @ down.T
    if kind == "experts":
        E, H, I = case["experts"], case["hidden"], case["inter"]
        gate_up, down = d.normal(E, 2 * I, H, std=0.02, dtype=dt), d.normal(E, H, I, std=0.02, dtype=dt)
        x = d.normal(case["rows"], H, dtype=dt).double()
        index, weight = _routing(case, d)
        out = torch.zeros_like(x)
        for e in range(E):
            row, slot = torch.where(index == e)
            if len(row):
                w = _stored(gate_up[e].float(), case["qtype"])
                a = torch.nn.functional.silu(x[row] @ w[:I].T) * (x[row] @ w[I:].T)
                out.index_add_(0, row, (a @ _stored(down[e].float(), case["qtype"]).T) * weight[row, slot, None].double())
        return out
    if kind == "train":
        w = _stored(_weight(d, case["n"], case["k"]), case["qtype"])
        x = d.normal(1, case["rows"], case["k"], dtype=dt).double()
        return x @ w.T, d.normal(1, case["rows"], case["n"], dtype=dt).double() @ w
    if kind == "attention":
        return _exact_attention(case, seed)
    if kind == "recurrence":
        return _exact_recurrence(case, seed)
    # step: the cache rounds keys and values to e5m2, a staircase that a run with other
    # low bits climbs elsewhere, so there is no 64-bit value that belongs to one run's logits
    return None
