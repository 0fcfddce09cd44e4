"""Performance cases of the quantised products: what a serving program has this package do.

Five kinds of work, through the package's public entry points:

  linear   one projection: a weight matrix in one of its formats times 1 .. 256 activation rows.
           One row is a decode step, a few rows are a speculative-decoding verifier batch, more
           are a prefill chunk.  f32 activations, or bf16 ones where an entry point takes them.
  layer    the projections of one decoder layer, each on what the one before wrote: q|k|v in one
           call, o, gate|up in one call, down -- what a decode loop launches per layer when it
           brings its own kernels for the rest.
  moe      one mixture-of-experts layer in MLX 4-bit: router, selected experts, weighted sum.
  experts  one mixture-of-experts layer over GGUF experts stacked in one matrix per projection:
           fused gate|up with GELU, then the weighted scatter-add of down, both by work list.
  generate greedy decoding with MLXDecoder: a prompt, then new tokens, the logits of the last one.

Shapes are those of the repository's benchmarks and tests (Llama-3 8B and 70B projections,
Qwen3-0.6B decoder, Qwen3-30B-A3B layer) and sizes between and around them.
"""
import math
import types

import numpy as np
import torch

from __graft_entry__ import load_package

PKG = load_package()
RT = PKG.runtime

# bytes per weight of the formats as their files store them
FILE_BYTES = {"mlx4": 0.5625, "q4_k": 144 / 256, "q5_k": 176 / 256, "q6_k": 210 / 256, "q8_0": 34 / 32, "fp8": 1.0}
GGUF_ID = {"q8_0": RT.GGUF_Q8_0, "q4_k": RT.GGUF_Q4_K, "q5_k": RT.GGUF_Q5_K, "q6_k": RT.GGUF_Q6_K}
# the matrices of this size and above are kept in the tensor-core layouts, which the bf16 entry points ask for
BIG = 8 << 20

DEC = types.SimpleNamespace(hidden=1024, layers=28, heads=16, kv_heads=8, head_dim=128, inter=3072, vocab=151936, eps=1e-6,
                            theta=1e6, qk_norm=True, max_seq=192)
DEC_SHAPES = {"q": (2048, 1024), "k": (1024, 1024), "v": (1024, 1024), "o": (1024, 2048), "gate": (3072, 1024),
              "up": (3072, 1024), "down": (1024, 3072)}


def _linear(name, fmt, out, inn, rows, x="f32"):
    return {"name": name, "op": "linear", "fmt": fmt, "out": out, "in": inn, "rows": rows, "x": x}


def _layer(name, hidden, q, kv, ffn, rows):
    return {"name": name, "op": "layer", "hidden": hidden, "q": q, "kv": kv, "ffn": ffn, "rows": rows}


def _experts_case(name, op, tokens, experts=128, top_k=8, hidden=2048, inter=768):
    return {"name": name, "op": op, "tokens": tokens, "experts": experts, "top_k": top_k, "hidden": hidden, "inter": inter}


def listed():
    return [
        # the smallest products of a decode step: a layer of a 0.6B model, where the launches are all there is
        _layer("decode layer mlx4 1024", 1024, 2048, 1024, 3072, 1),
        # the widest projection of an 8B model's decode step (gate|up stacked)
        _linear("decode mlx4 28672x4096", "mlx4", 28672, 4096, 1),
        # down projection of an 8B model in a Q4_K file
        _linear("decode q4_k 4096x14336", "q4_k", 4096, 14336, 1),
        # LM head of the same file: the K-quant mixes keep it in Q6_K
        _linear("decode q6_k 128256x4096", "q6_k", 128256, 4096, 1),
        # verifier batch of a 70B model in FP8, f32 activations
        _linear("verify fp8 8192x28672 x5", "fp8", 8192, 28672, 5),
        # attention output projection of an 8B model in Q8_0, a short ragged prefill chunk
        _linear("chunk q8_0 4096x4096 x19", "q8_0", 4096, 4096, 19),
        # gate projection of an 8B model in Q4_K, an ordinary prefill chunk
        _linear("prefill q4_k 14336x4096 x64", "q4_k", 14336, 4096, 64),
        # q|k|v of an 8B model in MLX 4-bit, f32 activations, an odd chunk
        _linear("prefill mlx4 6144x4096 x100", "mlx4", 6144, 4096, 100),
        # attention projection of a 70B model in MLX 4-bit, bf16 activations
        _linear("prefill mlx4 bf16 8192x8192 x64", "mlx4", 8192, 8192, 64, "bf16"),
        # gate|up of a 70B model in FP8, bf16 activations, the longest chunk: the largest product
        _linear("prefill fp8 bf16 28672x8192 x256", "fp8", 28672, 8192, 256, "bf16"),
        # an expert layer with eight tokens in flight (batched decode)
        _experts_case("moe mlx4 8 tokens", "moe", 8),
        # a whole small model: 63 steps, one token each
        {"name": "generate 32+32 tokens", "op": "generate", "prompt": 32, "new": 32},
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.random()
    case = _draw_one(rng, kind)
    case.pop("name", None)
    return case


def _draw_one(rng, kind):
    if kind < 0.18:
        return _experts_case(None, "moe" if kind < 0.1 else "experts", _log_int(rng, 1, 32), rng.choice([32, 64, 96, 128]), rng.randint(2, 8),
                             256 * rng.randint(4, 12), 256 * rng.randint(2, 6))
    if kind < 0.25:
        return {"op": "generate", "prompt": rng.randint(4, 32), "new": rng.randint(4, 32)}
    if kind < 0.35:
        kv = 128 * rng.randint(2, 8)
        return _layer(None, 256 * rng.randint(3, 16), kv * rng.choice([1, 2, 4]), kv, 256 * _log_int(rng, 8, 56), rng.choice([1, 1, 2, 4]))
    while True:
        fmt = rng.choice(["mlx4", "mlx4", "q4_k", "q4_k", "q8_0", "q6_k", "q5_k", "fp8", "fp8"])
        inn = 256 * _log_int(rng, 3, 112)
        if rng.random() < 0.2:  # widths that are no multiple of the K-quants' 256-element blocks
            if fmt in ("mlx4", "fp8"):
                inn += 64 * rng.randint(1, 3)
            elif fmt == "q8_0":
                inn += 32 * rng.randint(1, 7)
        out = _log_int(rng, 256, 28672)
        if rng.random() < 0.5:
            out = max(256, out // 256 * 256)
        r = rng.random()
        rows = 1 if r < 0.35 else rng.randint(2, 8) if r < 0.55 else _log_int(rng, 9, 256)
        bf16 = fmt in ("mlx4", "fp8") and rows > 1 and inn % 256 == 0 and out * inn >= BIG and rng.random() < 0.5
        if (4 << 20 if rows == 1 else 1 << 20) <= out * inn <= 28672 * 8192:
            return {"op": "linear", "fmt": fmt, "out": out, "in": inn, "rows": rows, "x": "bf16" if bf16 else "f32"}


# ---- inputs -------------------------------------------------------------------------------------

def _gen(seed, *more):
    g = torch.Generator(device="cuda")
    g.manual_seed(hash((seed,) + more) & 0x7FFFFFFF)
    return g


def _bytes(g, n):
    return torch.randint(0, 256, (n,), generator=g, device="cuda", dtype=torch.uint8)


def _uniform_f16_bytes(g, n, lo, hi):
    v = torch.rand(n, generator=g, device="cuda") * (hi - lo) + lo
    return v.to(torch.float16).view(torch.uint8).view(n, 2)


def _mlx_arrays(g, out, inn, zero=8.0):
    """Uniform nibbles; bf16 scales |N(0,1)| * 0.02 + 1e-3, bf16 biases -zero * scale (groups of 64)."""
    w = _bytes(g, out * inn // 2).cpu().numpy().view(np.uint32)
    s = (torch.randn(out * inn // 64, generator=g, device="cuda").abs() * 0.02 + 1e-3).to(torch.bfloat16).float()
    return w, s.cpu().numpy(), (-zero * s).to(torch.bfloat16).float().cpu().numpy()


def _gguf_bytes(g, fmt, out, inn):
    """Block bytes of a GGUF tensor: uniform quants and packed scales, f16 block scales in the files' range."""
    if fmt == "q8_0":
        n = out * (inn // 32)
        q = torch.randint(-127, 128, (n, 32), generator=g, device="cuda", dtype=torch.int8).view(torch.uint8)
        return torch.cat([_uniform_f16_bytes(g, n, 0.001, 0.02), q], 1).reshape(-1).cpu().numpy()
    n = out * (inn // 256)
    if fmt == "q6_k":
        sc = torch.randint(-127, 128, (n, 16), generator=g, device="cuda", dtype=torch.int8).view(torch.uint8)
        parts = [_bytes(g, n * 192).view(n, 192), sc, _uniform_f16_bytes(g, n, 0.0005, 0.005)]
    else:
        rest = {"q4_k": 140, "q5_k": 172}[fmt]
        parts = [_uniform_f16_bytes(g, n, 0.001, 0.02), _uniform_f16_bytes(g, n, 0.001, 0.02), _bytes(g, n * rest).view(n, rest)]
    return torch.cat(parts, 1).reshape(-1).cpu().numpy()


def _wrap(t):
    return RT.wrap(t.data_ptr(), t.numel() * t.element_size())


class _State:
    """What the program keeps between calls; its device memory goes back when it is dropped."""

    def __init__(self):
        self.owned = []

    def own(self, *handles):
        self.owned += handles
        return handles[0] if len(handles) == 1 else handles

    def __del__(self):
        try:
            for h in self.owned:
                h.Free()
        except Exception:  # the interpreter is going down
            pass


def _prepare_linear(case, seed):
    st, g = _State(), _gen(seed, 1)
    fmt, out, inn, rows = case["fmt"], case["out"], case["in"], case["rows"]
    if fmt == "mlx4":
        st.w = st.own(RT.UploadMLXWeight(*_mlx_arrays(g, out, inn), inn, out, 64, True))
    elif fmt == "fp8":
        w = torch.randn(out * inn, generator=g, device="cuda").clamp_(-448, 448).to(torch.float8_e4m3fn).view(torch.uint8)
        scale = (torch.rand(out, generator=g, device="cuda") * 1.5 + 0.5) / math.sqrt(inn)
        st.w = st.own(RT.UploadFP8E4M3Linear(w.cpu().numpy(), scale.cpu().numpy(), None, out, inn))
        del w
    else:
        st.w = st.own(RT.UploadGGUFMatrix(GGUF_ID[fmt], _gguf_bytes(g, fmt, out, inn), inn, out))
    x = torch.randn(rows, inn, generator=g, device="cuda")
    st.x = x.to(torch.bfloat16) if case["x"] == "bf16" or fmt == "mlx4" else x
    if case["x"] == "f32":
        st.x = st.x.float()  # MLX models hand on bf16 values in f32 buffers
    st.out = torch.zeros(rows, out, device="cuda")
    st.xb, st.yb, st.rows = _wrap(st.x), _wrap(st.out), rows
    if case["x"] == "bf16":
        st.call = _mlx_bf16 if fmt == "mlx4" else _fp8_bf16
    elif fmt == "mlx4":
        st.call = _mlx_gemv if rows == 1 else _mlx_gemm
    elif fmt == "fp8":
        st.call = _fp8_gemv if rows == 1 else _fp8_gemm
    else:
        st.call = _gguf
    return st


def _mlx_gemv(st):
    RT.GemvMLX(st.yb, st.xb, st.w)


def _mlx_gemm(st):
    RT.GemmMLX(st.yb, st.xb, st.w, st.rows)


def _mlx_bf16(st):
    RT.GemmMLXBF16(st.yb, st.xb, st.w, st.rows)


def _fp8_gemv(st):
    RT.GemvFP8E4M3Buffer(st.yb, st.xb, st.w)


def _fp8_gemm(st):
    RT.GemmFP8E4M3Buffer(st.yb, st.xb, st.rows, st.w)


def _fp8_bf16(st):
    RT.GemmFP8E4M3BF16Buffer(st.yb, st.xb, st.rows, st.w)


def _gguf(st):
    st.w.ProjectBatchToBuffer(st.yb, st.xb, st.rows)


def _prepare_layer(case, seed):
    st, g, rows = _State(), _gen(seed, 5), case["rows"]
    h, q, kv, f = case["hidden"], case["q"], case["kv"], case["ffn"]

    def weight(out, inn):  # zero-mean weights that keep the activations' size from product to product
        w, s, _ = _mlx_arrays(g, out, inn)
        s = (torch.from_numpy(s) / (0.08 * math.sqrt(inn))).to(torch.bfloat16).float()
        b = (-7.5 * s).to(torch.bfloat16).float()
        return st.own(RT.UploadMLXWeight(w, s.numpy(), b.numpy(), inn, out, 64, True))

    st.qkv, st.o = [weight(q, h), weight(kv, h), weight(kv, h)], weight(h, q)
    st.gu, st.down = [weight(f, h), weight(f, h)], weight(h, f)
    st.x = torch.randn(rows, h, generator=g, device="cuda").to(torch.bfloat16).float()
    st.out = {n: torch.zeros(rows, d, device="cuda") for n, d in (("q", q), ("k", kv), ("v", kv), ("o", h), ("gate", f), ("up", f), ("down", h))}
    st.buf = {n: _wrap(t) for n, t in st.out.items()}
    st.xb, st.rows = _wrap(st.x), rows
    st.call = _layer_step
    return st


def _layer_step(st):
    b = st.buf
    RT.GemmMLXMulti([b["q"], b["k"], b["v"]], st.xb, st.qkv, st.rows)
    RT.GemmMLX(b["o"], b["q"], st.o, st.rows)
    RT.GemmMLXMulti([b["gate"], b["up"]], b["o"], st.gu, st.rows)
    RT.GemmMLX(b["down"], b["gate"], st.down, st.rows)


def _prepare_moe(case, seed):
    """One token at a time is served from row-major experts, several from tiled ones (the layout is chosen at upload)."""
    st, g, tokens = _State(), _gen(seed, 2), case["tokens"]
    n, hidden, inter = case["experts"], case["hidden"], case["inter"]
    st.layer = RT.GPUMoELayer(n, hidden, inter, 64, case["top_k"], True, tokens)
    st.layer.SetRouter(st.own(RT.UploadMLXWeight(*_mlx_arrays(g, n, hidden), hidden, n, 64, True)))
    shapes = ((inter, hidden), (inter, hidden), (hidden, inter))
    host = [_mlx_arrays(g, n * o, i) for o, i in shapes]
    RT.SetOption("mlx_layout", 2 if tokens > 1 else 0)
    try:
        for e in range(n):
            three = []
            for (o, i), (w, s, b) in zip(shapes, host):
                nw, ns = o * i // 8, o * i // 64
                three.append(RT.UploadMLXWeight(w[e * nw:(e + 1) * nw], s[e * ns:(e + 1) * ns], b[e * ns:(e + 1) * ns], i, o, 64, True))
            st.layer.SetExpert(e, *st.own(*three))
    finally:
        RT.SetOption("mlx_layout", 0)
    st.own(st.layer)
    st.x = torch.randn(tokens, hidden, generator=g, device="cuda").to(torch.bfloat16).float()
    st.out = torch.zeros(tokens, hidden, device="cuda")
    st.xb, st.yb, st.tokens = _wrap(st.x), _wrap(st.out), tokens
    st.call = _moe
    return st


def _moe(st):
    st.layer.Forward(st.yb, st.xb, st.tokens)


def _prepare_experts(case, seed):
    st, g, tokens = _State(), _gen(seed, 3), case["tokens"]
    st.experts, hidden, st.inter = case["experts"], case["hidden"], case["inter"]
    rows_gu, rows_dn = st.experts * 2 * st.inter, st.experts * hidden
    st.gu = st.own(RT.UploadGGUFMatrix(RT.GGUF_Q4_K, _gguf_bytes(g, "q4_k", rows_gu, hidden), hidden, rows_gu))
    st.dn = st.own(RT.UploadGGUFMatrix(RT.GGUF_Q8_0, _gguf_bytes(g, "q8_0", rows_dn, st.inter), st.inter, rows_dn))
    k = case["top_k"]
    st.n = tokens * k
    st.ids = torch.rand(tokens, st.experts, generator=g, device="cuda").topk(k, 1).indices.to(torch.int32).reshape(-1).contiguous()
    st.pos = torch.arange(tokens, device="cuda", dtype=torch.int32).repeat_interleave(k).contiguous()
    st.wt = torch.rand(st.n, generator=g, device="cuda") * 0.15 + 0.05
    st.x = torch.randn(tokens, hidden, generator=g, device="cuda").repeat_interleave(k, 0).contiguous()  # a row per item
    st.act = torch.zeros(st.n, st.inter, device="cuda")
    st.out = torch.zeros(tokens, hidden, device="cuda")
    st.bufs = [_wrap(t) for t in (st.act, st.x, st.ids, st.out, st.pos, st.wt)]
    st.call = _experts
    return st


def _experts(st):
    act, x, ids, y, pos, wt = st.bufs
    y.Zero()
    RT.GateUpGELUQ4KByWorkToBuffer(act, x, ids, st.n, st.inter, st.experts, st.gu)
    RT.GemvQ8_0ScatterByWork(y, act, ids, pos, wt, st.n, st.experts, st.dn)


def _prepare_generate(case, seed):
    st, g, c = _State(), _gen(seed, 4), DEC
    # zero-mean weights (bias -7.5 scale), four distinct layers' worth of them in 28 device copies
    base = [{n: _mlx_arrays(g, o, i, 7.5) for n, (o, i) in DEC_SHAPES.items()} for _ in range(4)]

    def norm(n):
        return (1 + 0.1 * torch.randn(n, generator=g, device="cuda")).cpu().numpy()

    layers = [dict(base[l % 4], input_norm=norm(c.hidden), post_norm=norm(c.hidden), q_norm=norm(c.head_dim), k_norm=norm(c.head_dim))
              for l in range(c.layers)]
    ang = np.outer(np.arange(c.max_seq, dtype=np.float64), c.theta ** (-2.0 * np.arange(c.head_dim // 2) / c.head_dim))
    table = np.stack([np.cos(ang), np.sin(ang)], -1).astype(np.float32)
    st.dec = PKG.decode.MLXDecoder(RT, c, layers, _mlx_arrays(g, c.vocab, c.hidden, 7.5), norm(c.hidden), table)
    d = st.dec
    st.own(d.lm, d.final_norm, d.table, d.hidden, d.hidden2, d.normed, d.proj2, d.qkv, d.attn, d.proj, d.gu, d.act, d.logits, d.ints)
    for e in d.L:
        st.own(*[h for h in e.values() if h is not None])
    st.prompt = torch.randint(0, c.vocab, (case["prompt"],), generator=g, device="cuda").tolist()
    st.new = case["new"]
    d.reset(st.prompt)
    d.capture()  # once per model: the step's graph
    st.call = None
    return st


def _generate(st):
    tokens = st.dec.generate(st.prompt, st.new)
    return np.array(tokens, dtype=np.int64), st.dec.logits.Download()


_READY = False


def prepare(case, seed):
    global _READY
    if not _READY:
        RT.init(torch.cuda.current_device())
        _READY = True
    return {"linear": _prepare_linear, "layer": _prepare_layer, "moe": _prepare_moe, "experts": _prepare_experts,
            "generate": _prepare_generate}[case["op"]](case, seed)


def run(state):
    if state.call is None:
        return _generate(state)
    state.call(state)
    return state.out


# ---- what a pass cannot do without ---------------------------------------------------------------

def work(case):
    if case["op"] == "linear":
        o, i, m = case["out"], case["in"], case["rows"]
        b = o * i * FILE_BYTES[case["fmt"]] + (4 * o if case["fmt"] == "fp8" else 0) + m * i * (2 if case["x"] == "bf16" else 4) + 4 * m * o
        return {"bytes": b, "flops": 2 * o * i * m}
    if case["op"] == "layer":
        h, q, kv, f, m = case["hidden"], case["q"], case["kv"], case["ffn"], case["rows"]
        n = h * (2 * q + 2 * kv + 3 * f)
        return {"bytes": n * FILE_BYTES["mlx4"] + 4 * m * (5 * h + 2 * q + 2 * kv + 3 * f), "flops": 2 * n * m}
    if case["op"] == "generate":
        params = DEC.layers * sum(o * i for o, i in DEC_SHAPES.values()) + DEC.vocab * DEC.hidden
        steps = case["prompt"] + case["new"] - 1
        cache = DEC.layers * 2 * DEC.kv_heads * DEC.head_dim * 4 * steps * (steps + 1) / 2
        return {"bytes": steps * params * FILE_BYTES["mlx4"] + cache, "flops": 2 * steps * params}
    t, e, k, n = case["tokens"], case["experts"], case["top_k"], case["hidden"] * case["inter"]
    distinct = e * (1 - (1 - k / e) ** t)  # experts that the tokens of a call select, on average
    io = 8 * t * case["hidden"]
    if case["op"] == "moe":
        return {"bytes": distinct * 3 * n * FILE_BYTES["mlx4"] + e * case["hidden"] * FILE_BYTES["mlx4"] + io, "flops": 6 * n * t * k}
    per = 2 * n * FILE_BYTES["q4_k"] + n * FILE_BYTES["q8_0"]
    return {"bytes": distinct * per + io + 8 * t * k * case["inter"], "flops": 6 * n * t * k}


def tolerance(case):
    """Weights and activations are exact in every format and the sums are taken in f32, over up to 29k
    products in another order (and, for GPU sums in tensor-core accumulators, other groupings)."""
    if case["op"] == "generate":
        return {"rel": 1e-4, "max": 1e-3, "differ": 0.01}  # 28 layers of them, one behind the other
    if case["op"] == "linear":
        return {"rel": 2e-5, "max": 3e-4}
    return {"rel": 5e-5, "max": 1e-3}  # two to four products, one behind the other
