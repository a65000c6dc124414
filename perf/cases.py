"""What a program built on cera_b200 has it do, as cases that can be timed and checked.

Families: one quantized matrix times a column (`gemv`) or a batch of columns (`gemm`), decode attention over a long cache (`attend`), the
routed feed-forward (`moe`), and whole models through the model object: decoding on a resumed session (`llama_decode`), reading a
prompt (`llama_prompt`, `goletar_prompt`, `piditar_prompt`) and a short exchange - a prompt, then tokens one by one with the logits of
each in the caller's hands, as a sampler wants them (`goletar_session`, `piditar_session`).

Weights are random, quantized by the package's own quantizers where they are quantized; `exact` evaluates the same formulas in float64
with plain torch."""
import math

import numpy as np
import torch

import cera_b200 as cb
from cera_b200 import goletar, piditar, synth, types
from cera_b200.layered import Ff, LayeredModel, Mixer
from cera_b200.model import Role

QUANT = {"q4_0": types.Q4_0, "q4_1": types.Q4_1, "q8_0": types.Q8_0, "q4_k": types.Q4_K, "q5_k": types.Q5_K, "q6_k": types.Q6_K}
VOCAB = 32768
F64 = torch.float64


def listed():
    return [
        # the smallest call: one 4096 x 4096 Q4_0 projection of one token, activations quantized on the way
        dict(name="gemv_q4_0_4096", kind="gemv", type="q4_0", m=4096, k=4096),
        # a batch of 64 columns through the down projection of an 8B model: several short prompts at once, or a speculative batch
        dict(name="gemm_q6_k_down_64", kind="gemm", type="q6_k", m=4096, k=14336, n=64, image=False),
        # one decode step's attention over a long document held in f16
        dict(name="attend_f16_16384", kind="attend", heads=32, kv_heads=8, dim=128, context=16384, f16=True),
        # one token through a routed feed-forward layer: the decode step of a mixture-of-experts model
        dict(name="moe_q4_0_1", kind="moe", type="q4_0", experts=32, used=4, width=2048, ff=1792, n=1, softmax=False),
        # a prompt of 512 tokens through the same layer
        dict(name="moe_q4_0_512", kind="moe", type="q4_0", experts=32, used=4, width=2048, ff=1792, n=512, softmax=False),
        # the whole 8B-shape model answering at a context of 512: the step a chat user waits for
        dict(name="llama_decode_512", kind="llama_decode", width=4096, ff=14336, layers=32, vocab=128256, context=512, tokens=16, f16=False),
        # layers of the same model reading a prompt of one chunk
        dict(name="llama_prompt_512", kind="llama_prompt", width=4096, ff=14336, layers=2, vocab=128256, n=512, f16=False),
        # the same with a document that fills no chunk evenly, into an f16 cache
        dict(name="llama_prompt_2047", kind="llama_prompt", width=4096, ff=14336, layers=2, vocab=128256, n=2047, f16=True),
        # a long prompt of a model with latent attention, minGRU and routed experts
        dict(name="goletar_prompt_2048", kind="goletar_prompt", width=4096, layers=4, n=2048),
        # a question of a few lines and the first tokens of the answer
        dict(name="goletar_session_48", kind="goletar_session", width=2048, layers=4, n=48, tokens=16),
        # a long prompt of a model with grouped attention, real-gated and state-space recurrences
        dict(name="piditar_prompt_2048", kind="piditar_prompt", width=4096, layers=8, n=2048),
        # a longer question at the larger width, and the first tokens of the answer
        dict(name="piditar_session_200", kind="piditar_session", width=4096, layers=8, n=200, tokens=16),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["gemv", "gemm", "attend", "moe", "llama_decode", "llama_prompt", "goletar_prompt", "goletar_session", "piditar_prompt",
                       "piditar_session"])
    if kind in ("gemv", "gemm"):
        t = rng.choice(sorted(QUANT))
        unit = types.BLOCK[QUANT[t]][0]
        c = dict(kind=kind, type=t, m=_log(rng, 64, 14336), k=unit * max(1, _log(rng, 256, 14336) // unit))
        if kind == "gemm":
            c.update(n=_log(rng, 2, 2048), image=rng.random() < 0.5)
        return c
    if kind == "attend":
        heads, kv_heads = rng.choice([(32, 8), (32, 4), (8, 8), (16, 8), (24, 3)])
        return dict(kind=kind, heads=heads, kv_heads=kv_heads, dim=rng.choice([64, 128]), context=_log(rng, 16, 32768), f16=rng.random() < 0.5)
    if kind == "moe":
        return dict(kind=kind, type=rng.choice(["q4_0", "q4_0", "q8_0", "q4_k"]), experts=rng.choice([8, 16, 32]), used=rng.choice([2, 4]),
                    width=rng.choice([512, 1024, 2048]), ff=256 * rng.randint(1, 7), n=_log(rng, 1, 512), softmax=rng.random() < 0.5)
    if kind == "llama_decode":
        w = rng.choice([1024, 2048, 4096])
        return dict(kind=kind, width=w, ff=512 * rng.randint(w // 512, 7 * w // 1024), layers=rng.randint(2, 8), vocab=VOCAB, context=_log(rng, 16, 4096),
                    tokens=rng.randint(2, 16), f16=rng.random() < 0.5)
    if kind == "llama_prompt":
        w = rng.choice([1024, 2048, 4096])
        return dict(kind=kind, width=w, ff=512 * rng.randint(w // 512, 7 * w // 1024), layers=2, vocab=VOCAB, n=_log(rng, 32, 2047),
                    f16=rng.random() < 0.5)
    w = rng.choice([1024, 2048, 4096])
    if kind.endswith("prompt"):
        return dict(kind=kind, width=w, layers=4, n=_log(rng, 2, 2048))
    return dict(kind=kind, width=w, layers=4, n=_log(rng, 2, 600), tokens=rng.randint(2, 16))


# ---- inputs ----------------------------------------------------------------------------------------------------------

def _seed(seed, *what):
    """One generator seed out of a case's seed and a place in it."""
    h = seed & 0xFFFFFFFF
    for x in what:
        h = (h * 1000003 + int(x) + 0x9E3779B9) & 0x7FFFFFFFFFFFFFFF
    return h


def _normal(shape, *what, dtype=torch.float32):
    return torch.randn(shape, device="cuda", dtype=dtype, generator=torch.Generator("cuda").manual_seed(_seed(*what)))


def _tokens(n, vocab, seed):
    return torch.randint(0, vocab, (n,), generator=torch.Generator().manual_seed(_seed(seed, 77))).numpy().astype(np.uint32)


def _quantized(t, rows, cols, *what, sigma=0.02):
    """GGUF block bytes of a normal matrix, on the device."""
    return cb.quantize_weights(t, _normal(rows * cols, *what).mul_(sigma))


def _llama_tensors(case):
    """(role, layer, type, rows, cols) of every matrix: Q4_K throughout, Q6_K for the down projections and the head."""
    w, ff, kv = case["width"], case["ff"], case["width"] // 4
    yield Role.TOKEN_EMBD, 0, types.Q4_K, case["vocab"], w
    yield Role.OUTPUT, 0, types.Q6_K, case["vocab"], w
    for i in range(case["layers"]):
        for role, rows, cols in ((Role.ATTN_Q, w, w), (Role.ATTN_K, kv, w), (Role.ATTN_V, kv, w), (Role.ATTN_OUTPUT, w, w), (Role.FFN_GATE, ff, w),
                                 (Role.FFN_UP, ff, w), (Role.FFN_DOWN, w, ff)):
            yield role, i, types.Q6_K if role == Role.FFN_DOWN else types.Q4_K, rows, cols


def _llama_model(case, seed, max_seq_len):
    w = case["width"]
    model = cb.CudaModel(n_layers=case["layers"], hidden_size=w, intermediate_size=case["ff"], n_heads=w // 128, n_kv_heads=w // 512, head_dim=128,
                         vocab_size=case["vocab"], rope_theta=500000.0, rms_norm_eps=1e-5, rope_type=0, kv_f16=int(case["f16"]), max_seq_len=max_seq_len)
    for role, layer, t, rows, cols in _llama_tensors(case):
        model.add_tensor(role, layer, t, rows, cols, _quantized(t, rows, cols, seed, role, layer))
    ones = np.ones(w, dtype=np.float32)
    model.add_tensor(Role.OUTPUT_NORM, 0, types.F32, 1, w, ones)
    for i in range(case["layers"]):
        model.add_tensor(Role.ATTN_NORM, i, types.F32, 1, w, ones)
        model.add_tensor(Role.FFN_NORM, i, types.F32, 1, w, ones)
    torch.cuda.synchronize()
    model.finalize()
    return model


def _llama_cache(case, seed, layer):
    """Keys and values of a past conversation, of the size that unit-norm inputs and N(0, 0.02) weights give."""
    kv = [_normal((case["context"], case["width"] // 4), seed, 900 + i, layer).mul_(0.02 * math.sqrt(case["width"])) for i in (0, 1)]
    return [x.half() for x in kv] if case["f16"] else kv


def _layered_config(case):
    if case["kind"].startswith("goletar"):
        return goletar, synth.goletar_config(case["width"], case["layers"], vocab=VOCAB)
    return piditar, synth.piditar_config(case["width"], case["layers"], vocab=VOCAB)


def _layered_shape(role, d, width, buckets):
    """Rows and columns of a tensor of layer description d."""
    H, inner, n = d.n_heads, d.n_heads * d.value_dim, d.recurrent_width
    block = n // d.n_blocks if d.n_blocks else 0
    channels = inner + 2 * d.n_groups * d.state_size if d.mixer == Mixer.SSM else n
    latent, attention = d.mixer == Mixer.LATENT_ATTENTION, d.mixer in (Mixer.LATENT_ATTENTION, Mixer.ATTENTION, Mixer.SSM)
    norm = 1 if d.ff == Ff.MOE else width
    return {Role.TOKEN_EMBD: (VOCAB, width), Role.OUTPUT: (VOCAB, width), Role.BIGRAM_EMBD: (buckets + 1, width), Role.OUTPUT_NORM: (1, norm),
            Role.MIX_PRE_NORM: (1, norm), Role.MIX_POST_NORM: (1, norm), Role.FF_PRE_NORM: (1, norm), Role.FF_POST_NORM: (1, norm),
            Role.MIX_OUTPUT: (width, inner if attention else n), Role.LATENT_Q: (H * (d.head_dim + d.rot_dim), width),
            Role.LATENT_DOWN: (d.kv_rank + d.rot_dim, width), Role.LATENT_NORM: (1, d.kv_rank), Role.LATENT_UP_K: (H * d.head_dim, d.kv_rank),
            Role.LATENT_UP_V: (inner, d.kv_rank), Role.LATENT_SINK: (1, H), Role.LATENT_GATE: (H, width), Role.GRU_Z: (n, width), Role.GRU_X: (n, width),
            Role.GRU_GATE: (n, width), Role.GRU_Z_BIAS: (1, n), Role.GRU_X_BIAS: (1, n), Role.ROUTER: (d.n_experts, width),
            Role.EXPERT_GATE: (d.ff_width, width), Role.EXPERT_UP: (d.ff_width, width), Role.EXPERT_DOWN: (width, d.ff_width),
            Role.FFN_GATE: (d.ff_width, width), Role.FFN_UP: (d.ff_width, width), Role.FFN_DOWN: (width, d.ff_width),
            Role.ATTN_Q: (H * d.head_dim, width), Role.ATTN_K: (d.n_kv_heads * d.head_dim, width), Role.ATTN_V: (d.n_kv_heads * d.value_dim, width),
            Role.ATTN_Q_BIAS: (1, H * d.head_dim), Role.ATTN_K_BIAS: (1, d.n_kv_heads * d.head_dim), Role.ATTN_V_BIAS: (1, d.n_kv_heads * d.value_dim),
            Role.CONV: (channels, d.conv_taps), Role.CONV_BIAS: (1, channels), Role.LRU_OUT: (n, width), Role.LRU_IN: (n, width),
            Role.LRU_OUT_BIAS: (1, n), Role.LRU_IN_BIAS: (1, n), Role.LRU_DECAY_GATE: (n, block), Role.LRU_INPUT_GATE: (n, block),
            Role.LRU_DECAY_GATE_BIAS: (1, n), Role.LRU_INPUT_GATE_BIAS: (1, n), Role.LRU_LAMBDA: (1, n), Role.SSM_IN: (inner + channels + H, width),
            Role.SSM_DT_BIAS: (1, H), Role.SSM_A_LOG: (1, H), Role.SSM_D: (1, H), Role.SSM_NORM: (1, inner)}[role]


def _layered_value(case, seed, name, role, shape, place):
    """One bf16 tensor of a Goletar or Piditar model, of a scale that keeps every branch alive."""
    z = _normal(shape, seed, role, place, dtype=torch.bfloat16)
    leaf = name.rsplit(".", 1)[-1]
    if leaf.startswith("norm"):
        around = 1.0 if case["kind"].startswith("goletar") or role == Role.SSM_NORM else 0.0
        return z.mul_(0.3).add_(around)
    if leaf in ("embed", "bigram", "lam", "D"):
        return z
    if leaf == "sink":
        return z.add_(1.0)
    if leaf in ("dt_bias", "A_log"):
        return z.sub_(1.0)
    if leaf == "b":
        return z.mul_(0.5)
    return z.mul_((1.5 if leaf in ("gate", "up", "in", "x", "y", "z", "q") else 1.0) / math.sqrt(shape[1]))


def _layered_tensors(case, seed):
    """(name, role, layer, expert, maker of the tensor) of the model, in a fixed order."""
    design, config = _layered_config(case)
    buckets = config["embedding"].get("bigram", {}).get("buckets", 0)
    _, layers = design.describe(config)
    for place, (name, role, layer, expert) in enumerate(design.tensor_roles(layers)):
        shape = _layered_shape(role, layers[layer], case["width"], buckets)
        yield name, role, layer, expert, lambda n=name, r=role, s=shape, p=place: _layered_value(case, seed, n, r, s, p)


def _layered_model(case, seed, max_seq_len):
    design, config = _layered_config(case)
    kw, layers = design.describe(config)
    model = LayeredModel(layers, dtype="bfloat16", max_seq_len=max_seq_len, **kw)
    for _, role, layer, expert, make in _layered_tensors(case, seed):
        v = make()
        model.add_tensor(role, layer, types.BF16, v.shape[0], v.shape[1], v, expert=expert)
    torch.cuda.synchronize()
    model.finalize()
    return model


def _moe_inputs(case, seed):
    E, W, ff, t = case["experts"], case["width"], case["ff"], QUANT[case["type"]]
    return (_quantized(t, E * ff, W, seed, 1), _quantized(t, E * ff, W, seed, 2), _quantized(t, E * W, ff, seed, 3), _normal((E, W), seed, 4).mul_(0.05),
            _normal((case["n"], W), seed, 5))


def prepare(case, seed):
    kind = case["kind"]
    state = dict(case)
    if kind in ("gemv", "gemm"):
        t = QUANT[case["type"]]
        state["w"] = cb.QuantWeight(t, case["m"], case["k"], _quantized(t, case["m"], case["k"], seed, 1))
        if case.get("image"):
            state["w"].prepare_gemm()
        state["x"] = _normal(case.get("n", 1) * case["k"], seed, 2)
    elif kind == "attend":
        shape = (case["context"], case["kv_heads"] * case["dim"])
        half = torch.float16 if case["f16"] else torch.float32
        state.update(q=_normal(case["heads"] * case["dim"], seed, 1), kc=_normal(shape, seed, 2).to(half), vc=_normal(shape, seed, 3).to(half))
        need = cb.ops.lib.cera_cuda_decode_attention_workspace_bytes(case["heads"], case["dim"], case["context"])
        state["ws"] = torch.empty(need, dtype=torch.uint8, device="cuda")
    elif kind == "moe":
        gate, up, down, router, x = _moe_inputs(case, seed)
        state["ffn"] = cb.MoeFfn(case["experts"], case["used"], case["width"], case["ff"], QUANT[case["type"]], gate, up, down, router, max_tokens=512)
        state["x"] = x
    elif kind == "llama_decode":
        state["model"] = _llama_model(case, seed, case["context"] + case["tokens"] + 8)
        layers = [tuple(x.cpu().numpy().view(np.uint8).reshape(-1) for x in _llama_cache(case, seed, i)) for i in range(case["layers"])]
        state["model"].restore_state({"seq_len": case["context"], "layers": layers})
        state["toks"] = [int(t) for t in _tokens(2, case["vocab"], seed)]
    elif kind == "llama_prompt":
        state.update(model=_llama_model(case, seed, case["n"] + 8), toks=_tokens(case["n"], case["vocab"], seed))
    else:
        more = case.get("tokens", 0)
        state.update(model=_layered_model(case, seed, case["n"] + more + 8), toks=_tokens(case["n"] + more, VOCAB, seed))
    return state


def run(s):
    kind = s["kind"]
    if kind == "gemv":
        return cb.gemv(s["w"], s["x"])
    if kind == "gemm":
        return cb.gemm_preq(s["w"], cb.quantize_q8_0(s["x"], k=s["k"], n=s["n"]))
    if kind == "attend":
        return cb.decode_attention(s["q"], s["kc"], s["vc"], s["heads"], s["kv_heads"], s["dim"], s["context"], s["dim"] ** -0.5, workspace=s["ws"])
    if kind == "moe":
        out, ids, weights = s["ffn"](s["x"], softmax_gate=s["softmax"], want_routing=True)
        return {"out": out, "ids": ids, "weights": weights}
    model = s["model"]
    if kind == "llama_decode":
        model.truncate_kv(s["context"])
        logits = model.forward(s["toks"][0], s["context"])
        return {"logits": logits, "tokens": model.generate_greedy(s["toks"][1], s["context"] + 1, s["tokens"])[0]}
    model.truncate_kv(0)
    if kind.endswith("prompt"):
        return model.forward_prefill(s["toks"], 0)
    n = s["n"]
    return [model.forward_prefill(s["toks"][:n], 0)] + [model.forward(int(t), n + i) for i, t in enumerate(s["toks"][n:])]


# ---- what a pass cannot do without -----------------------------------------------------------------------------------

def _bytes(t, elements):
    per, size = types.BLOCK[t]
    return elements // per * size


def _layered_work(case):
    """(weight bytes of the layers that one token reads, of all experts, cached values of one position and run, elements of one token)."""
    design, config = _layered_config(case)
    _, layers = design.describe(config)
    fixed = expert = state = cache = 0
    for _, role, layer, e in design.tensor_roles(layers):
        d = layers[layer]
        rows, cols = _layered_shape(role, d, case["width"], 0)
        if role in (Role.TOKEN_EMBD, Role.BIGRAM_EMBD):
            continue
        if e is None:
            fixed += rows * cols
        else:
            expert += rows * cols
    if not case["kind"].startswith("goletar"):
        fixed += VOCAB * case["width"]  # the embedding is the head
    for d in layers:
        if d.mixer == Mixer.LATENT_ATTENTION:
            cache += d.kv_rank + d.rot_dim
        elif d.mixer == Mixer.ATTENTION:
            cache += d.n_kv_heads * (d.head_dim + d.value_dim)
        elif d.mixer == Mixer.SSM:
            state += d.n_heads * d.value_dim * d.state_size
        else:
            state += d.recurrent_width
    top = layers[0].n_used / layers[0].n_experts if layers[0].ff == Ff.MOE else 0
    attend = sum(2 * d.n_heads * (d.head_dim + d.rot_dim * (d.mixer == Mixer.LATENT_ATTENTION) + d.value_dim) for d in layers
                 if d.mixer in (Mixer.LATENT_ATTENTION, Mixer.ATTENTION))
    experts = layers[0].n_experts or 1
    return fixed, expert, top, experts, state, cache, attend


def work(case):
    kind, n = case["kind"], case.get("n", 1)
    if kind in ("gemv", "gemm"):
        m, k = case["m"], case["k"]
        return {"bytes": _bytes(QUANT[case["type"]], m * k) + 4 * n * (m + k), "flops": 2 * m * k * n}
    if kind == "attend":
        c = case["context"] * case["dim"]
        return {"bytes": c * case["kv_heads"] * 2 * (2 if case["f16"] else 4) + 8 * case["heads"] * case["dim"], "flops": 4 * c * case["heads"]}
    if kind == "moe":
        one = 3 * case["width"] * case["ff"]
        met = min(case["experts"], n * case["used"])
        return {"bytes": met * _bytes(QUANT[case["type"]], one) + 4 * case["experts"] * case["width"] + 8 * n * case["width"],
                "flops": 2 * n * (case["used"] * one + case["experts"] * case["width"])}
    if kind.startswith("llama"):
        w, L = case["width"], case["layers"]
        body = sum(_bytes(t, r * c) for role, _, t, r, c in _llama_tensors(case) if role not in (Role.TOKEN_EMBD, Role.OUTPUT))
        macs = sum(r * c for role, _, t, r, c in _llama_tensors(case) if role not in (Role.TOKEN_EMBD, Role.OUTPUT))
        head = _bytes(types.Q6_K, case["vocab"] * w)
        row = 2 * (w // 4) * (2 if case["f16"] else 4) * L  # one position's keys and values
        if kind == "llama_decode":
            steps, seen = case["tokens"] + 1, case["context"]
            return {"bytes": steps * (body + head + row * (seen + 1) + 4 * case["vocab"] // steps),
                    "flops": steps * (2 * macs + 2 * case["vocab"] * w + 4 * seen * w * L)}
        return {"bytes": body + head + row * n + 4 * case["vocab"], "flops": n * (2 * macs + 2 * n * w * L) + 2 * case["vocab"] * w}
    fixed, expert, top, experts, state, cache, attend = _layered_work(case)
    head = VOCAB * case["width"]

    def portion(m, before):
        share = 1 - (1 - top) ** m if top else 0
        return (2 * (fixed + expert * share) + 4 * state + 2 * cache * (before + m) + 4 * VOCAB,
                2 * m * (fixed - head + expert * top) + 2 * head + attend * m * (before + m / 2) + 6 * state * m)

    parts = [portion(n, 0)] + [portion(1, n + i) for i in range(case.get("tokens", 0))]
    return {"bytes": float(sum(b for b, _ in parts)), "flops": float(sum(f for _, f in parts))}


def tolerance(case):
    kind = case["kind"]
    if kind == "llama_decode":
        return "exact"  # the decode path evaluates one defined order of f32 operations
    if kind in ("gemv", "gemm"):
        return {"rel": 2e-6}  # f32 sums of exact products, in another order (measured against 64 bits: 4e-7)
    if kind == "attend":
        return {"rel": 1e-5}  # the same over 32768 positions (3e-6)
    if kind == "moe":
        return {"rel": 1e-3, "differ": 0.002}  # the gated unit is quantized to 8 bits again: one rounding moves a whole step (2e-4)
    if kind == "llama_prompt":
        return {"rel": 0.03, "max": 0.3}  # seven such quantizations a layer (2e-2; 1.2e-2 between two orders of the same sums)
    return {"rel": 0.03, "max": 0.3}  # bf16 products (1e-2)


# ---- the same in 64 bits -----------------------------------------------------------------------------------------------

def _half(raw, at):
    return raw[..., at:at + 2].contiguous().view(torch.float16).to(F64)


def _k_scales(raw):
    """The eight 6-bit scales and minima of Q4_K / Q5_K blocks."""
    s = raw[:, 4:16].to(torch.int16)
    low, high, mix = s[:, :4], s[:, 4:8], s[:, 8:]
    return (torch.cat([low & 63, (mix & 15) | ((low >> 6) << 4)], 1).to(F64), torch.cat([high & 63, (mix >> 4) | ((high >> 6) << 4)], 1).to(F64))


def _dequantized(t, raw, rows, cols):
    """The matrix that GGUF block bytes stand for."""
    elems, size = types.BLOCK[t]
    b = raw.view(-1, size)
    if t in (types.Q4_0, types.Q4_1):
        q = b[:, size - 16:]
        q = torch.cat([q & 15, q >> 4], 1).to(F64)
        w = _half(b, 0) * (q - 8) if t == types.Q4_0 else _half(b, 0) * q + _half(b, 2)
    elif t == types.Q8_0:
        w = _half(b, 0) * b[:, 2:].contiguous().view(torch.int8).to(F64)
    elif t in (types.Q4_K, types.Q5_K):
        sc, mn = _k_scales(b)
        q = b[:, size - 128:].view(-1, 4, 1, 32)
        q = torch.cat([q & 15, q >> 4], 2).reshape(-1, 8, 32)
        if t == types.Q5_K:
            bit = torch.arange(8, device=raw.device, dtype=torch.uint8).view(1, 8, 1)
            q = q + (((b[:, 16:48].view(-1, 1, 32) >> bit) & 1) << 4)
        w = (_half(b, 0) * sc).unsqueeze(2) * q.to(F64) - (_half(b, 2) * mn).unsqueeze(2)
    else:
        ql, qh = b[:, :128].view(-1, 2, 2, 32), b[:, 128:192].view(-1, 2, 1, 32)
        q = torch.cat([ql & 15, ql >> 4], 2) | (torch.cat([(qh >> s) & 3 for s in (0, 2, 4, 6)], 2) << 4)  # [block, half, group, 32]
        sc = b[:, 192:208].contiguous().view(torch.int8).to(F64).view(-1, 2, 4, 2, 1)
        w = _half(b, 208).view(-1, 1, 1, 1, 1) * sc * (q.to(F64) - 32).view(-1, 2, 4, 2, 16)
    return w.reshape(rows, cols)


def _q8(x):
    """Columns after their 8-bit quantization in blocks of 32 (f32 rules: scale amax / 127 kept in f16)."""
    v = x.to(torch.float32).view(*x.shape[:-1], -1, 32)
    d = v.abs().amax(-1, keepdim=True) / 127.0
    inv = torch.where(d > 0, 1.0 / d, torch.zeros_like(d))
    return (d.half().to(F64) * torch.round(v * inv).clamp(-128, 127).to(F64)).view(x.shape)


def _rms(x, eps, weight=1.0):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps) * weight


def _turned(x, start, base, dims):
    """Adjacent pairs of the first `dims` entries of the last axis turned by position; x: [T, heads, d]."""
    pos = torch.arange(start, start + x.shape[0], device=x.device, dtype=F64)
    a = pos[:, None] * torch.pow(torch.tensor(float(base), device=x.device, dtype=F64), -torch.arange(0, dims, 2, device=x.device, dtype=F64) / dims)
    c, s = torch.cos(a)[:, None], torch.sin(a)[:, None]
    u, v = x[..., 0:dims:2], x[..., 1:dims:2]
    return torch.cat([torch.stack([u * c - v * s, v * c + u * s], -1).flatten(-2), x[..., dims:]], -1)


def _attended(q, k, v, scale, cap=0.0, sink=None, q_rot=None, k_rot=None):
    """Causal attention of the last len(q) positions; q: [T, H, d], k, v: [S, G, d]; a shared rotated part beside it."""
    T, H, S, G = q.shape[0], q.shape[1], k.shape[0], k.shape[1]
    hidden = torch.arange(S, device=q.device)[None] > torch.arange(S - T, S, device=q.device)[:, None]
    out = []
    for h in range(H):
        g = h // (H // G)
        s = q[:, h] @ k[:, g].T
        if q_rot is not None:
            s = s + q_rot[:, h] @ k_rot.T
        s = s * scale
        if cap:
            s = cap * torch.tanh(s / cap)
        s = s.masked_fill(hidden, -math.inf)
        m = s.amax(-1, keepdim=True)
        if sink is not None:
            m = torch.maximum(m, sink[h])
        e = torch.exp(s - m)
        den = e.sum(-1, keepdim=True) + (torch.exp(sink[h] - m) if sink is not None else 0.0)
        out.append(e / den @ v[:, g])
    return torch.stack(out, 1)


def _exact_moe(case, seed):
    gate, up, down, router, x = _moe_inputs(case, seed)
    E, W, ff, t = case["experts"], case["width"], case["ff"], QUANT[case["type"]]
    s = x.to(F64) @ router.to(F64).T
    p = torch.softmax(s, -1) if case["softmax"] else torch.sigmoid(s)
    wt, ids = torch.sort(p, dim=-1, descending=True, stable=True)
    wt, ids = wt[:, :case["used"]], ids[:, :case["used"]]
    wt = wt / wt.sum(-1, keepdim=True).clamp_min(2.0 ** -14)
    out, xq = torch.zeros_like(x, dtype=F64), _q8(x)
    for e in range(E):
        tok, pick = torch.nonzero(ids == e, as_tuple=True)
        if not tok.numel():
            continue
        g, u, d = (_dequantized(t, m.view(E, -1)[e], r, c) for m, r, c in ((gate, ff, W), (up, ff, W), (down, W, ff)))
        h = torch.nn.functional.silu(xq[tok] @ g.T) * (xq[tok] @ u.T)
        out.index_add_(0, tok, wt[tok, pick][:, None] * (_q8(h) @ d.T))
    return {"out": out, "ids": None, "weights": wt}


def _exact_llama(case, seed, toks, start):
    """Logits of the last token."""
    W = case["width"]
    H, G = W // 128, W // 512
    known = {(role, layer): (t, r, c) for role, layer, t, r, c in _llama_tensors(case)}

    def raw(role, layer):
        t, r, c = known[role, layer]
        return t, _quantized(t, r, c, seed, role, layer), r, c

    def times(x, role, layer):
        return _q8(x) @ _dequantized(*raw(role, layer)).T

    t, b, _, _ = raw(Role.TOKEN_EMBD, 0)
    at = torch.from_numpy(np.asarray(toks, dtype=np.int64)).cuda()
    x = _dequantized(t, b.view(case["vocab"], -1)[at].contiguous(), len(toks), W)
    del b
    for i in range(case["layers"]):
        h = _rms(x, 1e-5)
        q = _turned(times(h, Role.ATTN_Q, i).view(-1, H, 128), start, 500000.0, 128)
        k = _turned(times(h, Role.ATTN_K, i).view(-1, G, 128), start, 500000.0, 128)
        v = times(h, Role.ATTN_V, i).view(-1, G, 128)
        if case["f16"]:
            k, v = k.half().to(F64), v.half().to(F64)
        if start:
            pk, pv = (c.to(F64).view(-1, G, 128) for c in _llama_cache(case, seed, i))
            k, v = torch.cat([pk, k]), torch.cat([pv, v])
        x = x + times(_attended(q, k, v, 128 ** -0.5).reshape(-1, W), Role.ATTN_OUTPUT, i)
        h = _rms(x, 1e-5)
        x = x + times(torch.nn.functional.silu(times(h, Role.FFN_GATE, i)) * times(h, Role.FFN_UP, i), Role.FFN_DOWN, i)
    h = _q8(_rms(x[-1:], 1e-5))
    t, b, rows, _ = raw(Role.OUTPUT, 0)
    step = 16384
    return torch.cat([(h @ _dequantized(t, b.view(rows, -1)[r:r + step].reshape(-1), min(step, rows - r), W).T)[0] for r in range(0, rows, step)])


def _conv(x, taps, bias):
    n = taps.shape[1]
    pad = torch.cat([torch.zeros(n - 1, x.shape[1], device=x.device, dtype=F64), x])
    return sum(pad[j:j + len(x)] * taps[:, j] for j in range(n)) + bias


def _exact_layered(case, seed, toks, rows):
    """Logits of the places `rows` of the sequence; None where bf16 can pick other experts than 64 bits do."""
    design, config = _layered_config(case)
    W, eps, T = case["width"], config["norm"]["eps"], len(toks)
    sure = torch.ones(T, dtype=torch.bool, device="cuda")
    made = {name: make for name, _, _, _, make in _layered_tensors(case, seed)}
    at = torch.from_numpy(np.asarray(toks, dtype=np.int64)).cuda()
    F = torch.nn.functional

    def w(name):
        v = made[name]().to(F64)
        return v[0] if v.shape[0] == 1 else v

    x = made["embed"]()[at].to(F64)
    if design is goletar:
        b = config["embedding"]["bigram"]
        row = (at[:-1] * b["mul_prev"] + at[1:] * b["mul_cur"]) % b["buckets"]
        x = x + made["bigram"]()[torch.cat([torch.tensor([b["buckets"]], device="cuda"), row])].to(F64)
        normed = lambda v, name: _rms(v, eps, w(name))  # noqa: E731
    else:
        x = x * config["embedding"]["scale"]
        normed = lambda v, name: _rms(v, eps, 1.0 + w(name))  # noqa: E731
    for i, entry in enumerate(config["layers"]):
        c, p, kind = entry["mixer"], f"l{i}.mix.", entry["type"]
        h = normed(x, f"l{i}.norm1")
        if kind == "latent_attention":
            H, d, r, rank = c["heads"], c["dim"], c["rot_dim"], c["kv_rank"]
            q, down = (h @ w(p + "q").T).view(T, H, d + r), h @ w(p + "dkv").T
            lat = _rms(down[:, :rank], eps, w(p + "dkv.norm"))
            y = _attended(q[..., :d], (lat @ w(p + "uk").T).view(T, H, d), (lat @ w(p + "uv").T).view(T, H, -1), c["scale"], sink=w(p + "sink"),
                          q_rot=_turned(q[..., d:], 0, c["rot"]["base"], r), k_rot=_turned(down[:, None, rank:], 0, c["rot"]["base"], r)[:, 0])
            y = (y * torch.sigmoid(h @ w(p + "g").T)[..., None]).reshape(T, -1)
        elif kind == "mingru":
            z, u = torch.sigmoid(h @ w(p + "z").T + w(p + "z.b")), h @ w(p + "x").T + w(p + "x.b")
            fed, s, y = z * torch.where(u >= 0, u + 0.5, torch.sigmoid(u)), torch.zeros(c["width"], device="cuda", dtype=F64), torch.empty_like(z)
            for t in range(T):
                s = torch.addcmul(fed[t], 1.0 - z[t], s)
                y[t] = s
            y = y * F.silu(h @ w(p + "g").T)
        elif kind == "attention":
            H, G, d = c["heads"], c["kv_heads"], c["dim"]
            q, k, v = ((h @ w(p + n).T + w(p + n + ".b")).view(T, m, -1) for n, m in (("q", H), ("k", G), ("v", G)))
            q, k = (_rms(_turned(a, 0, c["rot"]["base"], c["rot"]["dims"]), eps) for a in (q, k))
            y = _attended(q, k, v, c["scale"], cap=c["softcap"]).reshape(T, -1)
        elif kind == "rglru":
            B = c["blocks"]
            u = _conv(h @ w(p + "x").T + w(p + "x.b"), w(p + "conv"), w(p + "conv.b"))
            r, g = (torch.sigmoid(torch.einsum("tbi,boi->tbo", u.view(T, B, -1), w(p + n).view(B, c["width"] // B, -1)).reshape(T, -1) + w(p + n + ".b"))
                    for n in ("ra", "ri"))
            log_a = -8.0 * r * F.softplus(w(p + "lam"))
            a, fed = torch.exp(log_a), torch.sqrt(-torch.expm1(2.0 * log_a)) * g * u
            s, y = torch.zeros(c["width"], device="cuda", dtype=F64), torch.empty_like(u)
            for t in range(T):
                s = torch.addcmul(fed[t], a[t], s)
                y[t] = s
            y = y * F.gelu(h @ w(p + "y").T + w(p + "y.b"), approximate="tanh")
        else:
            H, P, N, G = c["heads"], c["vdim"], c["state"], c["groups"]
            z, xbc, dt = torch.split(h @ w(p + "in").T, [H * P, H * P + 2 * G * N, H], 1)
            u, b, cc = torch.split(F.silu(_conv(xbc, w(p + "conv"), w(p + "conv.b"))), [H * P, G * N, G * N], 1)
            u, b, cc = u.view(T, H, P), b.view(T, G, N).repeat_interleave(H // G, 1), cc.view(T, G, N).repeat_interleave(H // G, 1)
            dt = F.softplus(dt + w(p + "dt_bias"))
            a, s, y = torch.exp(-torch.exp(w(p + "A_log")) * dt), torch.zeros(H, N, P, device="cuda", dtype=F64), torch.empty(T, H, P, device="cuda", dtype=F64)
            for t in range(T):
                s = a[t, :, None, None] * s + (dt[t, :, None] * b[t])[:, :, None] * u[t][:, None]
                y[t] = torch.einsum("hnp,hn->hp", s, cc[t])
            y = (y + w(p + "D")[:, None] * u).view(T, -1) * F.silu(z)
            y = _rms(y.view(T, c["norm_groups"], -1), eps).view(T, -1) * w(p + "norm")
        y = y @ w(p + "o").T
        x = x + (normed(y, f"l{i}.norm1b") if design is goletar else y)
        h, p = normed(x, f"l{i}.norm2"), f"l{i}.mlp."
        if design is goletar:
            m, y = entry["mlp"], torch.zeros_like(x)
            s, ids = torch.sort(h @ w(p + "router").T, dim=-1, descending=True, stable=True)
            lim, top = m["expert"]["limit"], m["router"]["top"]
            wt = torch.sigmoid(s)
            sure &= s[:, top - 1] - s[:, top] > 0.05 * s.std(-1)
            for e in range(m["router"]["experts"]):
                tok, pick = torch.nonzero(ids[:, :top] == e, as_tuple=True)
                if tok.numel():
                    he = wt[tok, pick][:, None] * h[tok]
                    g, u = (he @ w(f"{p}e{e}.gate").T).clamp_max(lim), (he @ w(f"{p}e{e}.up").T).clamp(-lim, lim)
                    y.index_add_(0, tok, (g * torch.sigmoid(1.702 * g) * (u + 1.0)) @ w(f"{p}e{e}.down").T)
            x = x + normed(y, f"l{i}.norm2b")
        else:
            x = x + (F.silu(h @ w(p + "gate").T) * (h @ w(p + "up").T)) @ w(p + "down").T
    y = normed(x[rows], "final.norm") @ w("head" if design is goletar else "embed").T
    return [row if sure[at] else None for row, at in zip(y, rows)]


def exact(case, seed):
    kind = case["kind"]
    if kind in ("gemv", "gemm"):
        t, n = QUANT[case["type"]], case.get("n", 1)
        y = _dequantized(t, _quantized(t, case["m"], case["k"], seed, 1), case["m"], case["k"]) @ _q8(_normal(n * case["k"], seed, 2).view(n, -1)).T
        return y[:, 0] if kind == "gemv" else y
    if kind == "attend":
        s = prepare(case, seed)
        q, k, v = (s[a].to(F64).view(-1, h, case["dim"]) for a, h in (("q", case["heads"]), ("kc", case["kv_heads"]), ("vc", case["kv_heads"])))
        return _attended(q, k, v, case["dim"] ** -0.5).reshape(-1)
    if kind == "moe":
        return _exact_moe(case, seed)
    if kind == "llama_decode":
        return {"logits": _exact_llama(case, seed, _tokens(2, case["vocab"], seed)[:1], case["context"]), "tokens": None}
    if kind == "llama_prompt":
        return _exact_llama(case, seed, _tokens(case["n"], case["vocab"], seed), 0)
    n = case["n"]
    if kind.endswith("prompt"):
        return _exact_layered(case, seed, _tokens(n, VOCAB, seed), [n - 1])[0]
    return _exact_layered(case, seed, _tokens(n + case["tokens"], VOCAB, seed), list(range(n - 1, n + case["tokens"])))
