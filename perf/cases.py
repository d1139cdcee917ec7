"""The work that users of this framework have it do, as cases that can be timed and compared.

What the framework is used for: `quantize_` puts int4 or int8 weights into the linear layers of a language model, the model
then reads prompts (many activation rows per call) and decodes tokens (one row per sequence in the batch), and the other
model families of the framework run their sequence mixers as kernels behind the C interface.  The cases are single layers
and kernels of these paths, plus two whole calls of a shortened Llama model that return its logits.

Kinds of cases:
    linear      nn.Linear whose weight went through quantize_, called on [rows][in]: int4 (group sizes 32 to 256) and int8
    quantize    quantize_ on one weight: the int4 recipe, its HQQ search, or int8
    decode      DecodeEngine behind Generator (CUDA graph): tokens decoded one after the other for a batch of sequences
    prompt      the Transformer on one prompt over an empty cache
    attention   window attention over a prompt portion (the kernel of three model families), through the C interface
"""
import ctypes
import math

import torch
import torch.nn.functional as F

import torchao_fork_b200 as ao
from torchao_fork_b200 import _lib

DEV = "cuda"
_BF16 = 0   # AO_LM_BF16 of include/ao_b200_lm.h

# (out, in) of the linear layers of the repository's Llama configurations: 8B (also Mistral-7B), 3B, 70B
SHAPES = [(6144, 4096), (4096, 4096), (28672, 4096), (14336, 4096), (4096, 14336), (5120, 3072), (3072, 8192),
          (10240, 8192), (8192, 8192), (28672, 8192), (8192, 28672)]


def listed():
    return [
        # the smallest call: one layer of a decoded token, batch 1, eager; launch and host latency
        dict(name="linear int4 1 row", kind="linear", bits=4, group=128, rows=1, out=4096, inp=4096),
        # a served batch of 16 sequences through the up-projection of a 70B layer; bound by the weight's bytes
        dict(name="linear int4 16 rows", kind="linear", bits=4, group=128, rows=16, out=28672, inp=8192),
        # a short prompt or a batch of drafts: ragged row count, the finer of the common group sizes
        dict(name="linear int4 77 rows", kind="linear", bits=4, group=64, rows=77, out=14336, inp=4096),
        # a long prompt through an 8B up-projection; bound by the tensor cores
        dict(name="linear int4 2048 rows", kind="linear", bits=4, group=128, rows=2048, out=14336, inp=4096),
        # int8: a batch of 32 sequences, and a prompt of ragged length through a down-projection
        dict(name="linear int8 32 rows", kind="linear", bits=8, group=0, rows=32, out=8192, inp=8192),
        dict(name="linear int8 1000 rows", kind="linear", bits=8, group=0, rows=1000, out=4096, inp=14336),
        # preparing a model: the plain int4 recipe on the largest weight of a 70B layer, the HQQ search on an 8B weight
        dict(name="quantize int4", kind="quantize", recipe="int4", group=128, out=28672, inp=8192),
        dict(name="quantize hqq", kind="quantize", recipe="hqq", group=64, out=4096, inp=4096),
        # decoding: one sequence with int4 weights (the headline), a batch of eight with int8 weights
        dict(name="decode int4 1 sequence", kind="decode", model="Mistral-7B", layers=4, bits=4, group=128, batch=1, context=300, tokens=16),
        dict(name="decode int8 8 sequences", kind="decode", model="Mistral-7B", layers=4, bits=8, group=0, batch=8, context=300, tokens=16),
        # reading a prompt with the whole model
        dict(name="prompt int4 700 tokens", kind="prompt", model="Mistral-7B", layers=2, bits=4, group=128, tokens=700),
        # the attention of a prompt of 2048 tokens in a layer of the 2k-wide families
        dict(name="attention 2048 rows", kind="attention", rows=2048, past=0, heads=16, kv_heads=4, dim=128, maps=1, window=4096),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["linear"] * 7 + ["quantize"] * 2 + ["decode"] * 2 + ["prompt"] + ["attention"] * 2)
    if kind == "linear":
        bits = rng.choice([4, 4, 8])
        while True:
            rows = _log(rng, 1, 4096)
            out, inp = rng.choice(SHAPES)
            if rng.random() < 0.3:      # tensor-parallel shards, trimmed vocabularies: sizes off the powers of two
                out, inp = _log(rng, 1000, 20000), 256 * rng.randint(4, 56)
            if rows * out * inp <= 2048 * 14336 * 4096:
                return dict(kind=kind, bits=bits, group=rng.choice([32, 64, 128, 128, 256]) if bits == 4 else 0, rows=rows, out=out, inp=inp)
    if kind == "quantize":
        recipe = rng.choice(["int4", "int8", "hqq"])
        out, inp = rng.choice([s for s in SHAPES if recipe != "hqq" or s[0] * s[1] <= 4096 * 6144])
        if rng.random() < 0.5:
            out = rng.randint(out // 2, out)
        return dict(kind=kind, recipe=recipe, group=rng.choice([32, 64, 128, 256]) if recipe != "int8" else 0, out=out, inp=inp)
    if kind == "decode":
        bits = rng.choice([4, 8])
        return dict(kind=kind, model=rng.choice(["Mistral-7B", "13B"]), layers=rng.randint(1, 3), bits=bits,
                    group=rng.choice([64, 128]) if bits == 4 else 0, batch=rng.choice([1, 1, 2, 3, 5, 8, 16, 24, 32, 64]),
                    context=_log(rng, 16, 900), tokens=rng.randint(4, 16))
    if kind == "prompt":
        bits = rng.choice([4, 8])
        return dict(kind=kind, model="Mistral-7B", layers=rng.randint(1, 2), bits=bits, group=128 if bits == 4 else 0, tokens=_log(rng, 17, 900))
    heads, maps = rng.choice([8, 16, 32]), rng.choice([1, 1, 2])
    rows = _log(rng, 100, 2048)
    past = rng.choice([0, 0, rng.randint(1, 2048 - rows)]) if rows < 2000 else 0
    if heads == 32 and rows > 1400:
        heads = 16
    return dict(kind=kind, rows=rows, past=past, heads=heads, kv_heads=rng.choice([2, 4, 8]), dim=128 // maps, maps=maps, window=rng.choice([512, 4096]))


# ------------------------------------------------------------------------------------------------ inputs
def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _weight(case, gen):
    """Weights of a trained linear layer: near normal, a spread of row scales."""
    w = torch.randn(case["out"], case["inp"], generator=gen, device=DEV)
    return (w * (0.02 * torch.exp(0.3 * torch.randn(case["out"], 1, generator=gen, device=DEV)))).to(torch.bfloat16)


def _rows(case, gen):
    """Activations behind a norm: near normal, a few channels larger than the others."""
    x = torch.randn(case["rows"], case["inp"], generator=gen, device=DEV)
    return (x * torch.exp(0.5 * torch.randn(1, case["inp"], generator=gen, device=DEV))).to(torch.bfloat16)


def _config(recipe, group):
    if recipe in (8, "int8"):
        return ao.Int8WeightOnlyConfig()
    return ao.Int4WeightOnlyConfig(group_size=group, use_hqq=recipe == "hqq")


def _module(w):
    lin = torch.nn.Linear(1, 1, bias=False, device="meta", dtype=torch.bfloat16)
    lin.out_features, lin.in_features = w.shape
    lin.weight = torch.nn.Parameter(w, requires_grad=False)
    return lin


def _args(case):
    from torchao_fork_b200._models.llama.model import ModelArgs
    cfg = ModelArgs.from_name(case["model"])
    cfg.n_layer = case["layers"]
    return cfg


def _weights(case, gen):
    """The parameters of the shortened model by their names, bf16."""
    from torchao_fork_b200._models.llama.model import Transformer
    with torch.device("meta"):
        model = Transformer(_args(case))
    out = {}
    for name, p in model.named_parameters():
        if p.dim() == 1:
            out[name] = (1 + 0.1 * torch.randn(p.shape, generator=gen, device=DEV)).to(torch.bfloat16)
        else:
            std = 1.0 if "embeddings" in name else p.shape[1] ** -0.5
            out[name] = torch.randn(p.shape, generator=gen, device=DEV, dtype=torch.bfloat16).mul_(std)
    return model, out


def _model(case, gen):
    model, weights = _weights(case, gen)
    model.load_state_dict(weights, assign=True)
    model = model.eval().requires_grad_(False)
    ao.quantize_(model, _config(case["bits"], case["group"]))
    return model


def _tokens(case, gen, *shape):
    return torch.randint(0, _args(case).vocab_size, shape, generator=gen, device=DEV)


def _cached(case, gen, cfg):
    """Keys and values of the context: [layer] -> (k, v), each [batch][kv heads][context][head size]."""
    shape = (case["batch"], cfg.n_local_heads, case["context"], cfg.head_dim)
    return [tuple(torch.randn(shape, generator=gen, device=DEV, dtype=torch.bfloat16) for _ in range(2)) for _ in range(cfg.n_layer)]


def _attention_inputs(case, gen):
    n, past, H, G, d, maps = (case[k] for k in ("rows", "past", "heads", "kv_heads", "dim", "maps"))
    q = torch.randn(n, H, maps, d, generator=gen, device=DEV) * 1.5
    k, v = (torch.randn(past + n, G, w, generator=gen, device=DEV, dtype=torch.bfloat16) for w in (maps * d, 128))
    return q, k, v


def prepare(case, seed):
    gen = _gen(seed)
    kind = case["kind"]
    if kind == "linear":
        lin = _module(_weight(case, gen))
        ao.quantize_(lin, _config(case["bits"], case["group"]))
        return dict(kind=kind, lin=lin, x=_rows(case, gen))
    if kind == "quantize":
        return dict(kind=kind, w=_weight(case, gen), config=_config(case["recipe"], case["group"]), int8=case["recipe"] == "int8")
    if kind == "decode":
        from torchao_fork_b200._models.llama.generate import Generator
        model = _model(case, gen)
        cfg, B, ctx, T = model.config, case["batch"], case["context"], case["tokens"]
        g = Generator(model, B, ctx + T, temperature=0.0)
        for blk, (k, v) in zip(model.layers, _cached(case, gen, cfg)):
            blk.attention.kv_cache.k_cache[:, :, :ctx] = k
            blk.attention.kv_cache.v_cache[:, :, :ctx] = v
        return dict(kind=kind, engine=g.engine, generator=g, context=ctx, tokens=_tokens(case, gen, T, B))
    if kind == "prompt":
        model = _model(case, gen)
        T = case["tokens"]
        model.setup_caches(1, T, device=torch.device(DEV))
        return dict(kind=kind, model=model, tokens=_tokens(case, gen, 1, T), pos=torch.arange(T, device=DEV, dtype=torch.int32))
    # attention: one sequence, its first `past` positions in the ring, the others brought by this step
    n, past, H, G, d, maps = (case[k] for k in ("rows", "past", "heads", "kv_heads", "dim", "maps"))
    q, k, v = _attention_inputs(case, gen)
    ring = max(case["window"], past + n)
    ring_k = torch.zeros(1, ring, G * maps * d, dtype=torch.bfloat16, device=DEV)
    ring_v = torch.zeros(1, ring, G * 128, dtype=torch.bfloat16, device=DEV)
    ring_k[0, :past], ring_v[0, :past] = k[:past].flatten(1), v[:past].flatten(1)
    rows = ctypes.c_int()
    _lib.lm_check(_lib.lm().ao_lm_window_attention_prompt_plan(_BF16, maps, H, G, d, 128, ctypes.byref(rows)), "window_attention_prompt_plan")
    first = torch.arange(0, n, rows.value, dtype=torch.int32)
    i32 = lambda t: t.to(torch.int32).to(DEV)  # noqa: E731
    back = torch.arange(n)
    return dict(kind=kind, q=q, k=k[past:].contiguous(), v=v[past:].contiguous(), ring_k=ring_k, ring_v=ring_v, ring=ring, slot=i32(back * 0),
                pos=i32(back + past), back=i32(back), first=i32(first), count=i32((n - first).clamp(max=rows.value)), case=dict(case),
                out=torch.empty(n, H * 128, dtype=torch.bfloat16, device=DEV))


# ------------------------------------------------------------------------------------------------ one pass
@torch.no_grad()
def run(state):
    kind = state["kind"]
    if kind == "linear":
        return state["lin"](state["x"])
    if kind == "quantize":
        lin = _module(state["w"])
        ao.quantize_(lin, state["config"])
        impl = lin.weight.tensor_impl
        return [impl.packed, impl.scale] if state["int8"] else [impl.packed_weight, impl.scale_and_zero]
    if kind == "decode":
        # the tokens are given (a continuation is scored), so that a near tie between two tokens changes nothing that follows
        eng, tokens = state["engine"], state["tokens"]
        eng.set_state(tokens[0], state["context"])
        eng.step()
        for t in tokens[1:]:
            eng.tok.copy_(t)
            eng.step()
        return eng.logits
    if kind == "prompt":
        return state["model"](state["tokens"], state["pos"])
    s, c = state, state["case"]
    _lib.lm_check(_lib.lm().ao_lm_window_attention_prompt(
        s["q"].data_ptr(), s["k"].data_ptr(), s["v"].data_ptr(), s["ring_k"].data_ptr(), s["ring_v"].data_ptr(), None, None, s["ring"], 0, _BF16,
        s["slot"].data_ptr(), s["pos"].data_ptr(), s["back"].data_ptr(), s["first"].data_ptr(), s["count"].data_ptr(), s["first"].numel(), c["maps"],
        c["heads"], c["kv_heads"], c["dim"], 128, c["window"], 0, c["dim"] ** -0.5, 0.4 if c["maps"] == 2 else 0.0, int(c["maps"] == 2), 1e-6, 1.0,
        s["out"].data_ptr(), s["out"].stride(0), torch.cuda.current_stream().cuda_stream), "window_attention_prompt")
    return s["out"]


# ------------------------------------------------------------------------------------------------ floors
def _weight_bytes(bits, group, n, k):
    return n * k / 2 + k // group * n * 4 if bits == 4 else n * k + 2 * n


def _layer_shapes(cfg):
    d, kv = cfg.dim, cfg.n_local_heads * cfg.head_dim
    return [(d + 2 * kv, d), (d, d), (2 * cfg.intermediate_size, d), (d, cfg.intermediate_size)]


def _pairs(case):
    """(query, key) pairs inside the window."""
    return sum(min(case["past"] + i + 1, case["window"]) for i in range(case["rows"]))


def work(case):
    kind = case["kind"]
    if kind == "linear":
        m, n, k = case["rows"], case["out"], case["inp"]
        return {"bytes": _weight_bytes(case["bits"], case["group"], n, k) + 2 * m * (n + k), "flops": 2 * m * n * k}
    if kind == "quantize":
        n, k = case["out"], case["inp"]
        return {"bytes": 2 * n * k + _weight_bytes(8 if case["recipe"] == "int8" else 4, case["group"], n, k), "flops": 0}
    if kind == "attention":
        n, H, G, d, maps = (case[k] for k in ("rows", "heads", "kv_heads", "dim", "maps"))
        keys = min(case["past"] + n, n + case["window"])
        return {"bytes": n * H * (maps * d * 4 + 256) + keys * G * (maps * d + 128) * 2, "flops": 2 * _pairs(case) * H * maps * (d + 128)}
    cfg = _args(case)
    shapes = _layer_shapes(cfg) * cfg.n_layer + [(cfg.vocab_size, cfg.dim)]
    weights = sum(_weight_bytes(case["bits"], case["group"], n, k) for n, k in shapes)
    params = sum(n * k for n, k in shapes)
    kv = 4 * cfg.n_layer * cfg.n_local_heads * cfg.head_dim      # bytes of one position's keys and values
    if kind == "decode":
        rows, T = case["batch"], case["tokens"]
        seen = sum(case["context"] + t + 1 for t in range(T))
        return {"bytes": T * (weights + 2 * rows * (cfg.dim + cfg.vocab_size)) + rows * kv * seen,
                "flops": 2 * T * rows * params + 4 * rows * seen * cfg.n_layer * cfg.dim}
    T = case["tokens"]
    return {"bytes": weights + 2 * T * (cfg.dim + cfg.vocab_size) + T * kv, "flops": 2 * T * params + 2 * T * (T + 1) * cfg.n_layer * cfg.dim}


def tolerance(case):
    kind = case["kind"]
    if kind == "quantize":
        # whole numbers and parameters are defined bit for bit; HQQ iterates in 32 bits, where the order of a group's sum can
        # move a value across a rounding boundary
        return {"rel": 1e-3, "max": 0.1, "differ": 1e-3} if case["recipe"] == "hqq" else "exact"
    if kind == "decode":
        return {"rel": 4e-2, "max": 0.4}    # bf16 residual stream and cache through every layer
    if kind == "prompt":
        return {"rel": 4e-2, "max": 0.6}
    # bf16 results, 32-bit sums; int4 weights rounded to bf16 or not in front of the product, int8 results rounded twice
    return {"rel": 1e-2, "max": 0.1}


# ------------------------------------------------------------------------------------------------ the same in 64 bits
def _int4_params(w, group):
    """The int4 recipe on bf16 weights as its definition rounds it -> whole numbers 0 .. 15, scale, zero, [out][groups][...]."""
    g = w.reshape(w.shape[0], -1, group)
    lo, hi = g.amin(-1, keepdim=True), g.amax(-1, keepdim=True)
    scale = ((hi - lo) / 15).clamp(min=1e-6)
    zero = lo + scale * 8
    q = ((g - (zero - scale * 8)) / scale).round().clamp(0, 15)
    return q, scale, zero


def _dequantized(w, bits, group):
    """The quantized weight as float64 [out][in]."""
    if bits == 4:
        q, scale, zero = _int4_params(w, group)
        return ((q.double() - 8) * scale.double() + zero.double()).reshape(w.shape)
    q, scale = _int8_params(w)
    return q.double() * scale.double()


def _int8_params(w):
    scale = (w.abs().amax(1, keepdim=True) / 127.5).clamp(min=torch.finfo(torch.float32).eps)
    return (w * (1.0 / scale)).round().clamp(-128, 127), scale


def _strips(scale, zero):
    """[out][groups] -> the stored order [out / 16][groups][16][2], rows padded to 128 with zeros."""
    s = torch.stack([scale, zero], -1)
    s = F.pad(s, (0, 0, 0, 0, 0, -s.shape[0] % 128))
    return s.reshape(s.shape[0] // 16, 16, s.shape[1], 2).permute(0, 2, 1, 3).contiguous()


def _hqq(w, group):
    g = w.double().reshape(w.shape[0], -1, group)
    lo, hi = g.amin(-1, keepdim=True), g.amax(-1, keepdim=True)
    scale = (15 / (hi - lo)).clamp(max=2e4)
    zero = (-lo * scale).round()
    best, beta = 1e4, 10.0
    for _ in range(20):
        q = (g * scale + zero).round().clamp(0, 15)
        diff = g - (q - zero) / scale
        e = diff.sign() * (diff.abs() - diff.abs().pow(-0.3) / beta).clamp(min=0)
        zero = (q - (g - e) * scale).mean(-1, keepdim=True)
        beta *= 1.01
        err = float(diff.abs().mean())
        if err >= best:
            break
        best = err
    return ((1 / scale).squeeze(-1), ((8 - zero) / scale).squeeze(-1))


def _llama(case, weights, x, freqs, past=None):
    """The Llama blocks on embedded rows x [batch][tokens][dim] in float64; `past`: cached keys and values per layer."""
    cfg = _args(case)
    B, T, _ = x.shape
    H, G, d = cfg.n_head, cfg.n_local_heads, cfg.head_dim
    W = lambda name: _dequantized(weights[name], case["bits"], case["group"])  # noqa: E731
    norm = lambda v, name: v * torch.rsqrt(v.square().mean(-1, keepdim=True) + cfg.norm_eps) * weights[name].double()  # noqa: E731

    def turn(v):
        p = v.reshape(B, T, -1, d // 2, 2)
        c, s = freqs[:, 0].view(1, T, 1, -1), freqs[:, 1].view(1, T, 1, -1)
        return torch.stack([p[..., 0] * c - p[..., 1] * s, p[..., 1] * c + p[..., 0] * s], -1).reshape(B, T, -1, d).transpose(1, 2)

    for i in range(cfg.n_layer):
        at, ff = f"layers.{i}.attention.", f"layers.{i}.feed_forward."
        q, k, v = (norm(x, f"layers.{i}.attention_norm.weight") @ W(at + "wqkv.weight").t()).split([H * d, G * d, G * d], -1)
        q, k, v = turn(q), turn(k), v.reshape(B, T, G, d).transpose(1, 2)
        P = 0
        if past is not None:
            k, v = (torch.cat([c.double(), new], 2) for c, new in zip(past[i], (k, v)))
            P = case["context"]
        k, v = k.repeat_interleave(H // G, 1), v.repeat_interleave(H // G, 1)
        s = q @ k.transpose(-1, -2) * d ** -0.5
        hidden = torch.arange(P + T, device=DEV)[None, :] > torch.arange(P, P + T, device=DEV)[:, None]
        y = (s.masked_fill(hidden, -math.inf).softmax(-1) @ v).transpose(1, 2).reshape(B, T, -1)
        x = x + y @ W(at + "wo.weight").t()
        h = norm(x, f"layers.{i}.ffn_norm.weight")
        x = x + (F.silu(h @ W(ff + "w1.weight").t()) * (h @ W(ff + "w3.weight").t())) @ W(ff + "w2.weight").t()
    return norm(x, "norm.weight"), W("output.weight")


def _angles(cfg, first, count):
    f = 1.0 / (cfg.rope_base ** (torch.arange(0, cfg.head_dim, 2, device=DEV).double() / cfg.head_dim))
    a = torch.outer(torch.arange(first, first + count, device=DEV).double(), f)
    return torch.stack([a.cos(), a.sin()], 1)


@torch.no_grad()
def exact(case, seed):
    gen = _gen(seed)
    kind = case["kind"]
    if kind == "linear":
        w = _weight(case, gen)
        x = _rows(case, gen).double()
        step = max(1, (1 << 27) // case["inp"])
        return torch.cat([x @ _dequantized(w[i : i + step], case["bits"], case["group"]).t() for i in range(0, case["out"], step)], 1)
    if kind == "quantize":
        w = _weight(case, gen)
        if case["recipe"] == "int8":
            return [None, (w.double().abs().amax(1) / 127.5).clamp(min=torch.finfo(torch.float32).eps)]
        if case["recipe"] == "hqq":
            scale, zero = _hqq(w, case["group"])
        else:
            g = w.double().reshape(w.shape[0], -1, case["group"])
            scale = ((g.amax(-1) - g.amin(-1)) / 15).clamp(min=1e-6)
            zero = g.amin(-1) + 8 * scale
        return [None, _strips(scale, zero)]
    if kind == "attention":
        q, k, v = (t.double() for t in _attention_inputs(case, gen))
        n, past, H, G, d, maps = (case[key] for key in ("rows", "past", "heads", "kv_heads", "dim", "maps"))
        i, j = torch.arange(past, past + n, device=DEV)[:, None], torch.arange(past + n, device=DEV)[None, :]
        hidden = (j > i) | (i - j >= case["window"])
        out = []
        for h in range(H):
            g = h // (H // G)
            maps_out = [(q[:, h, m] @ k[:, g, m * d : (m + 1) * d].t() * d ** -0.5).masked_fill(hidden, -math.inf).softmax(-1) @ v[:, g]
                        for m in range(maps)]
            y = maps_out[0]
            if maps == 2:
                y = y - 0.4 * maps_out[1]
                y = y * torch.rsqrt(y.square().mean(-1, keepdim=True) + 1e-6)
            out.append(y)
        return torch.cat(out, 1)
    cfg = _args(case)
    _, weights = _weights(case, gen)
    emb = weights["tok_embeddings.weight"]
    if kind == "decode":
        past, T = _cached(case, gen, cfg), case["tokens"]
        tokens = _tokens(case, gen, T, case["batch"])
        x, out = _llama(case, weights, emb[tokens.t()].double(), _angles(cfg, case["context"], T), past)
        return x[:, -1] @ out.t()
    tokens = _tokens(case, gen, 1, case["tokens"])
    x, out = _llama(case, weights, emb[tokens].double(), _angles(cfg, 0, case["tokens"]))
    return x @ out.t()
