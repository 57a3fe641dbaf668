"""Performance cases: the work a program gives this framework, through its public entry points.

A case is a dict of plain values.  Kinds:

  linear     `layers.Linear` of one quantisation type: what the operator API serves
  head       `ops.dense_gemm_skinny` with fp32 logits: the vocabulary projection of a decode step
  mlp_w4     gate/up projection with the SwiGLU epilogue and the down projection with the residual epilogue, 4-bit weights
  experts    the two grouped products of a mixture of experts, rows routed to several experts each
  attention  `ops.decode_attention`: one token per task over ragged caches, or a portion of a prompt under a causal mask
  decode     one step of `LlamaDecoder` for a batch of tasks, host tokens in, logits out (4-bit weights)
  prompt     `LlamaDecoder.prefill` of one prompt in portions, logits of its last position out (4-bit weights)
"""
import math

import numpy as np
import torch

from zhilight_b200 import layers, ops
from zhilight_b200.llama import LlamaDecoder

GROUP = 128                                   # quantisation group of the 4-bit weights
NORMAL, INT8, GPTQ, FP8 = layers.QUANT_NONE, layers.QUANT_INT8, layers.QUANT_GPTQ, layers.QUANT_FP8
MODEL = dict(num_layers=2, dim_model=4096, num_heads=32, num_kv_heads=8, dim_head=128, dim_ff=14336, vocab_size=32000, eps=1e-5,
             rope_theta=500000.0)             # the layers of an 8-billion-parameter Llama, two of them, a 32000-word vocabulary
PORTION = 512                                 # rows of a prompt per step, the engine's usual step size
MODEL_SEQ = 2048


def listed():
    return [
        # one token of one user through an attention output projection, 4-bit weights: latency counts
        dict(name="linear_w4_one_token", kind="linear", quant=GPTQ, m=1, k=4096, n=4096, bias=False),
        # 24 users decoding at once, 8-bit integer weights and activations, a biased projection
        dict(name="linear_int8_batch", kind="linear", quant=INT8, m=24, k=8192, n=8192, bias=True),
        # part of a prompt through an 8-bit floating-point feed-forward projection
        dict(name="linear_fp8_prompt", kind="linear", quant=FP8, m=500, k=4096, n=14336, bias=False),
        # a prompt through an unquantised feed-forward projection of a 1-billion-parameter Llama
        dict(name="linear_bf16_prompt", kind="linear", quant=NORMAL, m=777, k=2048, n=8192, bias=False),
        # the vocabulary projection of eight decoding users
        dict(name="head_bf16", kind="head", m=8, k=4096, n=128256),
        # the feed-forward of 32 decoding users and of a long prompt's portion, 4-bit weights
        dict(name="mlp_w4_batch", kind="mlp_w4", m=32, d=4096, f=14336),
        dict(name="mlp_w4_prompt", kind="mlp_w4", m=1000, d=4096, f=14336),
        # the experts of a portion of a prompt: 16 experts, four of them for every row
        dict(name="experts_prompt", kind="experts", tokens=512, width=2048, ff=2048, experts=16, top=4),
        # 32 users decoding over caches of different lengths
        dict(name="attention_decode", kind="attention", dtype="f16", batch=32, len_q=1, ctx=4096, heads=32, kv_heads=8, dim=128),
        # a portion of a prompt behind a thousand cached positions
        dict(name="attention_prompt", kind="attention", dtype="bf16", batch=1, len_q=500, ctx=1500, heads=32, kv_heads=8, dim=128),
        # whole calls: a step of four users, and the prompt of one
        dict(name="decode_step", kind="decode", batch=4, ctx=300),
        dict(name="prompt_1100", kind="prompt", tokens=1100),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["linear", "linear", "linear", "head", "mlp_w4", "mlp_w4", "experts", "attention", "attention", "attention", "decode",
                       "prompt"])
    if kind == "linear":
        quant = rng.choice([NORMAL, INT8, GPTQ, FP8])
        k = 128 * _log(rng, 8, 64)
        n = 32 * _log(rng, 16, 448)
        m = _log(rng, 1, 1024)
        return dict(kind=kind, quant=quant, m=max(1, min(m, (1 << 22) // k)), k=k, n=n, bias=rng.random() < 0.3)
    if kind == "head":
        return dict(kind=kind, m=_log(rng, 1, 32), k=256 * rng.randint(4, 16), n=8 * _log(rng, 2000, 16032))
    if kind == "mlp_w4":
        return dict(kind=kind, m=_log(rng, 1, 1000), d=128 * rng.randint(8, 32), f=128 * rng.randint(16, 112))
    if kind == "experts":
        experts = rng.choice([8, 16, 32])
        return dict(kind=kind, tokens=_log(rng, 1, 512), width=128 * rng.randint(4, 16), ff=64 * rng.randint(8, 32), experts=experts,
                    top=rng.choice([1, 2, 4]))
    if kind == "attention":
        heads, kv_heads, dim = rng.choice([(32, 8, 128), (32, 8, 64), (16, 16, 64), (8, 1, 128), (64, 8, 128), (16, 4, 128)])
        if rng.random() < 0.5:
            batch, len_q, ctx = _log(rng, 1, 32), 1, _log(rng, 17, 4096)
        else:
            len_q = _log(rng, 9, 512)
            batch, ctx = 1, len_q + rng.choice([0, _log(rng, 1, 1024)])
        return dict(kind=kind, dtype=rng.choice(["f16", "bf16"]), batch=batch, len_q=len_q, ctx=ctx, heads=heads, kv_heads=kv_heads, dim=dim)
    if kind == "decode":
        return dict(kind=kind, batch=_log(rng, 1, 16), ctx=_log(rng, 2, 500))
    return dict(kind=kind, tokens=_log(rng, 9, 1100))


# ---- inputs --------------------------------------------------------------------------------------------------------------------
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _randn(g, *shape, dtype=torch.float32, scale=1.0):
    return (torch.randn(*shape, generator=g, device="cuda") * scale).to(dtype)


def _gptq(g, k, n, spread=1.0):
    """A 4-bit projection as checkpoints hold it: words of eight rows, zeros minus one in words of eight columns, fp16 scales."""
    words = torch.randint(-2 ** 31, 2 ** 31, (k // 8, n), generator=g, device="cuda", dtype=torch.int64).to(torch.int32)
    zeros = torch.randint(6, 9, (k // GROUP, n // 8, 8), generator=g, device="cuda", dtype=torch.int64)
    shift = torch.arange(0, 32, 4, device="cuda")
    z = (zeros << shift).sum(-1)
    z = torch.where(z >= 2 ** 31, z - 2 ** 32, z).to(torch.int32)
    scales = ((0.5 + torch.rand(k // GROUP, n, generator=g, device="cuda")) * (0.2 * spread / k ** 0.5)).half()
    return {"qweight": words, "qzeros": z, "scales": scales}


def _gptq_matrix(t):
    """The (k, n) matrix that _gptq's tensors stand for, in 64 bits."""
    shift = torch.arange(0, 32, 4, device="cuda", dtype=torch.int32)
    q = (t["qweight"][:, None, :] >> shift[None, :, None]) & 15
    q = q.reshape(-1, t["qweight"].shape[1])
    z = (((t["qzeros"][:, :, None] >> shift) & 15) + 1) & 15
    z = z.reshape(t["qzeros"].shape[0], -1)
    return (q.double() - z.double().repeat_interleave(GROUP, 0)) * t["scales"].double().repeat_interleave(GROUP, 0)


def _linear_tensors(case, g):
    k, n, quant = case["k"], case["n"], case["quant"]
    if quant == GPTQ:
        t = _gptq(g, k, n)
    elif quant == INT8:
        t = {"weight": torch.randint(-127, 128, (n, k), generator=g, device="cuda", dtype=torch.int8),
             "weight_scale": (0.5 + torch.rand(n, generator=g, device="cuda")) * (0.014 / k ** 0.5)}
    elif quant == FP8:
        t = {"weight": _randn(g, n, k, scale=60.0).clamp(-448, 448).to(torch.float8_e4m3fn).view(torch.uint8),
             "weight_scale": torch.tensor([1 / (60.0 * k ** 0.5)], device="cuda")}
    else:
        t = {"weight": _randn(g, n, k, scale=k ** -0.5)}
    if case["bias"]:
        t["bias"] = _randn(g, n, scale=0.3)
    dtype = torch.float16 if quant in (GPTQ, INT8) else torch.bfloat16
    return t, _randn(g, case["m"], k, dtype=dtype), dtype


def _mlp_tensors(case, g):
    d, f = case["d"], case["f"]
    return _gptq(g, d, f), _gptq(g, d, f), _gptq(g, f, d, spread=2.0), _randn(g, case["m"], d, dtype=torch.float16), \
        _randn(g, case["m"], d, dtype=torch.float16)


def _packed(t, row_map=None):
    km = ops.gptq_to_k_major(t["qweight"], t["qzeros"], t["scales"])
    return ops.w4_pack(*km, GROUP, row_map=row_map, variant=1)


def _expert_tensors(case, g):
    """Rows, weights (gate and up rows in turn) and the routing lists a router leaves: rows sorted by expert."""
    t, d, f, e, top = (case[x] for x in ("tokens", "width", "ff", "experts", "top"))
    x = _randn(g, t, d, dtype=torch.bfloat16)
    up = _randn(g, e, 2 * f, d, dtype=torch.bfloat16, scale=d ** -0.5)
    down = _randn(g, e, d, f, dtype=torch.bfloat16, scale=f ** -0.5)
    liking = _randn(g, e) * 0.5 - torch.log(-torch.log(torch.rand(t, e, generator=g, device="cuda").clamp(1e-7, 1 - 1e-7)))
    chosen = liking.topk(top, dim=1).indices.reshape(-1)             # some experts are liked more than others
    order = torch.sort(chosen, stable=True).indices
    offsets = torch.zeros(e + 1, dtype=torch.int32, device="cuda")
    offsets[1:] = torch.bincount(chosen, minlength=e).cumsum(0).to(torch.int32)
    return x, up, down, offsets, (order // top).to(torch.int32), order.to(torch.int32)


def _lens(case):
    """Cache lengths of the tasks: from the longest down to a quarter of it."""
    b, ctx = case["batch"], case["ctx"]
    return [max(1, ctx - (3 * ctx * i) // (4 * b)) for i in range(b)]


def _attention_tensors(case, g):
    dtype = torch.float16 if case["dtype"] == "f16" else torch.bfloat16
    lens, hk, d = _lens(case), case["kv_heads"], case["dim"]
    q = _randn(g, case["batch"], case["len_q"], case["heads"], d, dtype=dtype, scale=1.5)
    ks = [_randn(g, n, hk, d, dtype=dtype) for n in lens]
    vs = [_randn(g, n, hk, d, dtype=dtype) for n in lens]
    mask = None
    if case["len_q"] > 1:                                            # row i of the portion sees the positions up to its own
        n, m = case["ctx"], case["len_q"]
        mask = (torch.arange(n, device="cuda")[None, :] <= torch.arange(n - m, n, device="cuda")[:, None]).to(torch.int8).contiguous()
    return q, ks, vs, mask, lens


def _model_tensors(g):
    c = MODEL
    d, f, hd, kd = c["dim_model"], c["dim_ff"], c["num_heads"] * c["dim_head"], c["num_kv_heads"] * c["dim_head"]
    t = {"token_embedding.weight": _randn(g, c["vocab_size"], d, dtype=torch.float16, scale=0.5),
         "lm_head.weight": _randn(g, c["vocab_size"], d, dtype=torch.float16, scale=d ** -0.5),
         "output_layernorm.weight": (1 + _randn(g, d, scale=0.1)).half()}
    shapes = {"attn.project_q": (d, hd), "attn.project_k": (d, kd), "attn.project_v": (d, kd), "attn.attn_out": (hd, d), "ff.w_in": (d, f),
              "ff.w_gated": (d, f), "ff.w_out": (f, d)}
    for i in range(c["num_layers"]):
        p = "layers.%d." % i
        for name in ("ln_attn", "ln_ff"):
            t[p + name + ".weight"] = (1 + _randn(g, d, scale=0.1)).half()
        for name, (k, n) in shapes.items():
            for part, v in _gptq(g, k, n).items():
                t[p + name + "." + part] = v
    return t


def _model_tokens(case, seed):
    rng = np.random.default_rng(seed)
    if case["kind"] == "prompt":
        return rng.integers(0, MODEL["vocab_size"], case["tokens"]).astype(np.int32)
    lens = _lens(case)
    return [rng.integers(0, MODEL["vocab_size"], n + 1).astype(np.int32) for n in lens]


def prepare(case, seed):
    g, kind = _gen(seed), case["kind"]
    if kind == "linear":
        t, x, dtype = _linear_tensors(case, g)
        lin = layers.Linear(case["k"], case["n"], "", case["quant"], "half" if dtype == torch.float16 else "bfloat")
        lin.load_state_dict(t)
        return {"kind": kind, "linear": lin, "x": x}
    if kind == "head":
        return {"kind": kind, "w": _randn(g, case["n"], case["k"], dtype=torch.bfloat16, scale=case["k"] ** -0.5),
                "x": _randn(g, case["m"], case["k"], dtype=torch.bfloat16)}
    if kind == "mlp_w4":
        gate, up, down, x, res = _mlp_tensors(case, g)
        both = {name: torch.cat([gate[name], up[name]], dim=1).contiguous() for name in gate}
        return {"kind": kind, "gate_up": _packed(both, ops.swiglu_row_map(case["f"], x.device)), "down": _packed(down), "x": x, "residual": res,
                "d": case["d"], "f": case["f"]}
    if kind == "experts":
        x, up, down, offsets, rows, pairs = _expert_tensors(case, g)
        return {"kind": kind, "x": x, "up": up, "down": down, "offsets": offsets, "rows": rows, "pairs": pairs}
    if kind == "attention":
        q, ks, vs, mask, lens = _attention_tensors(case, g)
        return {"kind": kind, "q": q, "k": ks, "v": vs, "mask": mask, "lens": torch.tensor(lens, dtype=torch.int32, device="cuda"),
                "longest": max(lens), "kv_heads": case["kv_heads"], "scale": case["dim"] ** -0.5}
    batch = case["batch"] if kind == "decode" else 1
    dec = LlamaDecoder(quant_type=GPTQ, group_size=GROUP, dtype="f16", max_batch=batch, max_seq=MODEL_SEQ, prefill_chunk=PORTION, **MODEL)
    dec.load_state_dict({name: t.cpu().numpy() for name, t in _model_tensors(g).items()})
    tokens = _model_tokens(case, seed)
    if kind == "prompt":
        return {"kind": kind, "model": dec, "tokens": tokens}
    for i, t in enumerate(tokens):
        dec.prefill(i, t[:-1], 0)
    return {"kind": kind, "model": dec, "tokens": np.array([t[-1] for t in tokens], dtype=np.int32),
            "positions": np.array([len(t) - 1 for t in tokens], dtype=np.int32)}


# ---- one pass ------------------------------------------------------------------------------------------------------------------
def run(s):
    kind = s["kind"]
    if kind == "linear":
        return s["linear"](s["x"])
    if kind == "head":
        return ops.dense_gemm_skinny(s["x"], s["w"], out_dtype=torch.float32)
    if kind == "mlp_w4":
        d, f = s["d"], s["f"]
        act = ops.w4a16_gemm_fused(s["x"], s["gate_up"], 2 * f, d, GROUP, epilogue=ops.EPI_SWIGLU, variant=1)
        return ops.w4a16_gemm_fused(act, s["down"], d, f, GROUP, residual=s["residual"], epilogue=ops.EPI_RESIDUAL, variant=1)
    if kind == "experts":
        n = s["rows"].numel()
        act = ops.gemm_nt_grouped(s["x"], s["up"], s["offsets"], n, x_rows=s["rows"], epilogue=ops.GEMM_EPI_GLU_CLAMP, limit=7.0, alpha=1.702,
                                  beta=1.0)
        return ops.gemm_nt_grouped(act, s["down"], s["offsets"], n, y_rows=s["pairs"], out_dtype=torch.float32)
    if kind == "attention":
        return ops.decode_attention(s["q"], s["lens"], s["k"], s["v"], s["mask"], s["scale"], s["longest"], s["kv_heads"])
    if kind == "decode":
        return s["model"].decode(s["tokens"], s["positions"], want_logits=True)[1]
    return s["model"].prefill(0, s["tokens"], 0, want_logits=True)[1]


# ---- what a pass cannot do without ---------------------------------------------------------------------------------------------
W4_BYTES = 0.5 + 2.5 / GROUP                  # a 4-bit weight with its share of the group's fp16 scale and 4-bit zero


def work(case):
    kind = case["kind"]
    if kind == "linear":
        m, k, n = case["m"], case["k"], case["n"]
        each = {GPTQ: W4_BYTES, INT8: 1, FP8: 1, NORMAL: 2}[case["quant"]]
        return {"bytes": n * k * each + 2 * m * (k + n) + 2 * n * (case["bias"] + (case["quant"] == INT8)), "flops": 2 * m * k * n}
    if kind == "head":
        m, k, n = case["m"], case["k"], case["n"]
        return {"bytes": 2 * n * k + 2 * m * k + 4 * m * n, "flops": 2 * m * k * n}
    if kind == "mlp_w4":
        m, d, f = case["m"], case["d"], case["f"]
        return {"bytes": 3 * d * f * W4_BYTES + 2 * m * 3 * d, "flops": 6 * m * d * f}
    if kind == "experts":
        t, d, f, e, top = (case[x] for x in ("tokens", "width", "ff", "experts", "top"))
        used = e * (1 - (1 - top / e) ** t)                          # experts that get a row
        return {"bytes": used * 3 * d * f * 2 + t * d * 2 + t * top * d * 4, "flops": t * top * 6 * d * f}
    if kind == "attention":
        lens, d, h = _lens(case), case["dim"], case["heads"]
        m, n = case["len_q"], case["ctx"]
        pairs = sum(lens) if m == 1 else sum(n - m + 1 + i for i in range(m))
        masked = m * n if m > 1 else 0
        return {"bytes": sum(lens) * case["kv_heads"] * d * 4 + case["batch"] * m * h * d * 4 + masked, "flops": 4 * pairs * h * d}
    c = MODEL
    d, f, hd, kd = c["dim_model"], c["dim_ff"], c["num_heads"] * c["dim_head"], c["num_kv_heads"] * c["dim_head"]
    weights = c["num_layers"] * (d * (hd + 2 * kd) + hd * d + 3 * d * f)
    rows = case["batch"] if kind == "decode" else 1
    before = sum(n + 1 for n in _lens(case)) if kind == "decode" else 0
    tokens = rows if kind == "decode" else case["tokens"]
    pairs = before if kind == "decode" else tokens * (tokens + 1) // 2
    cached = before if kind == "decode" else tokens
    return {"bytes": weights * W4_BYTES + 2 * c["vocab_size"] * d + 4 * rows * c["vocab_size"] + c["num_layers"] * cached * kd * 4 + 2 * tokens * d,
            "flops": 2 * tokens * weights + 2 * rows * d * c["vocab_size"] + c["num_layers"] * 4 * pairs * hd}


def tolerance(case):
    """About four times the distance from the same sums in 64 bits: the output's rounding, the rounding of 4-bit weights to fp16 and of
    probabilities, and in whole calls the fp16 residual stream."""
    kind = case["kind"]
    if kind == "head":
        return {"rel": 1e-5}
    if kind == "experts":
        return {"rel": 7e-3}
    if kind in ("decode", "prompt"):
        return {"rel": 2e-3}
    half = case["dtype"] == "f16" if kind == "attention" else kind == "mlp_w4" or case["quant"] in (GPTQ, INT8)
    return {"rel": 2e-3 if half else 7e-3}


# ---- the same in 64 bits -------------------------------------------------------------------------------------------------------
def _attend(q, k, v, visible, scale):
    """q (m, h, d), k and v (n, hk, d) in 64 bits, visible (m, n) or None -> (m, h, d)."""
    m, h, d = q.shape
    hk = k.shape[1]
    out = torch.empty_like(q)
    for j in range(hk):
        heads = slice(j * (h // hk), (j + 1) * (h // hk))
        s = torch.einsum("mhd,nd->hmn", q[:, heads], k[:, j]) * scale
        if visible is not None:
            s = s.masked_fill(~visible[None], -math.inf)
        out[:, heads] = torch.einsum("hmn,nd->mhd", torch.softmax(s, -1), v[:, j])
    return out


def _exact_linear(case, seed):
    t, x, dtype = _linear_tensors(case, _gen(seed))
    quant = case["quant"]
    if quant == GPTQ:
        y = x.double() @ _gptq_matrix(t)
    elif quant == INT8:                                              # the 8-bit rows are part of what the layer is
        top = x.float().abs().amax(1, keepdim=True)
        q = torch.round(x.float() * (127.0 / top))
        y = (q.double() @ t["weight"].double().T) * (top / 127.0).double() * t["weight_scale"].to(dtype).double()
    elif quant == FP8:
        scale = x.float().abs().amax() / 448.0
        q = (x.float() * (1.0 / scale)).half().float().to(torch.float8_e4m3fn)
        y = (q.double() @ t["weight"].view(torch.float8_e4m3fn).double().T) * (scale.double() * t["weight_scale"].double())
    else:
        y = x.double() @ t["weight"].to(dtype).double().T
    return y + t["bias"].to(dtype).double() if case["bias"] else y


def _exact_model(case, seed):
    c = MODEL
    t = _model_tensors(_gen(seed))
    h, hk, d, eps = c["num_heads"], c["num_kv_heads"], c["dim_head"], c["eps"]
    tokens = _model_tokens(case, seed)
    tokens = tokens if case["kind"] == "decode" else [tokens]

    def norm(x, w):
        return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + eps) * w.double()

    def turn(x, n):
        f = c["rope_theta"] ** (-torch.arange(0, d, 2, device="cuda", dtype=torch.float64) / d)
        a = torch.arange(n, device="cuda", dtype=torch.float64)[:, None, None] * f
        lo, hi = x[..., :d // 2], x[..., d // 2:]
        return torch.cat([lo * a.cos() - hi * a.sin(), hi * a.cos() + lo * a.sin()], -1)

    xs = [t["token_embedding.weight"][torch.from_numpy(x.astype(np.int64)).cuda()].double() for x in tokens]
    for i in range(c["num_layers"]):
        p = "layers.%d." % i
        w = {name: _gptq_matrix({part: t[p + name + "." + part] for part in ("qweight", "qzeros", "scales")})
             for name in ("attn.project_q", "attn.project_k", "attn.project_v", "attn.attn_out", "ff.w_in", "ff.w_gated", "ff.w_out")}
        for b, x in enumerate(xs):
            n = x.shape[0]
            a = norm(x, t[p + "ln_attn.weight"])
            q, k, v = ((a @ w["attn.project_" + y]).view(n, -1, d) for y in "qkv")
            seen = torch.ones(n, n, device="cuda").tril().bool()
            x = x + _attend(turn(q, n), turn(k, n), v, seen, d ** -0.5).reshape(n, -1) @ w["attn.attn_out"]
            a = norm(x, t[p + "ln_ff.weight"])
            xs[b] = x + (torch.nn.functional.silu(a @ w["ff.w_in"]) * (a @ w["ff.w_gated"])) @ w["ff.w_out"]
    last = torch.stack([x[-1] for x in xs])
    return norm(last, t["output_layernorm.weight"]) @ t["lm_head.weight"].double().T


def exact(case, seed):
    kind = case["kind"]
    if kind == "linear":
        return _exact_linear(case, seed)
    if kind in ("decode", "prompt"):
        return _exact_model(case, seed)
    if kind == "head":
        s = prepare(case, seed)
        return torch.cat([s["x"].double() @ w.double().T for w in s["w"].split(16384)], 1)
    g = _gen(seed)
    if kind == "mlp_w4":
        gate, up, down, x, res = _mlp_tensors(case, g)
        x = x.double()
        return (torch.nn.functional.silu(x @ _gptq_matrix(gate)) * (x @ _gptq_matrix(up))) @ _gptq_matrix(down) + res.double()
    if kind == "experts":
        x, up, down, offsets, rows, pairs = _expert_tensors(case, g)
        out = torch.zeros(rows.numel(), case["width"], dtype=torch.float64, device="cuda")
        bounds = offsets.tolist()
        for e in range(case["experts"]):
            part = slice(bounds[e], bounds[e + 1])
            h = x[rows[part].long()].double() @ up[e].double().T
            a, u = h[:, 0::2].clamp(max=7.0), h[:, 1::2].clamp(-7.0, 7.0)
            out[pairs[part].long()] = (a * torch.sigmoid(1.702 * a) * (u + 1.0)) @ down[e].double().T
        return out
    q, ks, vs, mask, _ = _attention_tensors(case, g)
    return torch.stack([_attend(q[b].double(), ks[b].double(), vs[b].double(), None if mask is None else mask.bool(), case["dim"] ** -0.5)
                        for b in range(case["batch"])])
