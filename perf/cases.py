"""Performance cases: the work a user of this package has it do, through its public entry points.

Five kinds of work:

stack   a batch of requests through ``DecodeStack``: the prompts are taken in, then tokens are decoded greedily, and the
        host reads the emitted tokens.  What a serving loop does; everything between is one CUDA graph per token.
layer   one decoder layer issued call by call through the launchers, as a host executor drives the C ABI: norm + quant,
        QKV with RoPE and the paged KV write, attention, O, norm + quant, gate|up with activation, down.
gemm    the four projections of a layer on M rows of FP8 activations: decode batches, speculative or chunked rows, prefill.
attn    paged FP8 decode attention over ragged contexts, sliding-window and global.
rows    the row kernels on T tokens: residual add + norm + quant, quant, activation + quant, RoPE + KV write, argmax.
"""
import math

import torch

from rvllm_b200 import ACT_GELU_TANH, ACT_SILU, BF16, F16, gemm, launchers, stack
from rvllm_b200.attention import PagedDecodeFp8Launcher, PagedDecodeParams

# Layer dimensions: the 31B-class benchmark shape, the CPU-checkable single-layer shape, and two generic ones in between
# (grouped-query with four query heads per KV head; a small one whose sizes are no multiples of the larger tiles).
DIMS = {
    "31b": dict(hidden=5376, ffn=21504, vocab=262144, heads=32, kv_heads=16, head_dim=128, global_head_dim=256, window=1024),
    "tiny": dict(hidden=512, ffn=2048, vocab=2048, heads=8, kv_heads=4, head_dim=64, global_head_dim=64, window=64),
    "mid": dict(hidden=4096, ffn=14336, vocab=128256, heads=32, kv_heads=8, head_dim=128, global_head_dim=128, window=1024),
    "small": dict(hidden=1152, ffn=3456, vocab=32000, heads=8, kv_heads=4, head_dim=128, global_head_dim=256, window=512),
}
DTYPES = {"f16": (F16, torch.float16), "bf16": (BF16, torch.bfloat16)}
ACTS = {"silu": ACT_SILU, "gelu": ACT_GELU_TANH}
EPS = 1e-6
PAGE = 16
ARGMAX_ROWS = 64  # a step samples at most so many sequences at once in the `rows` cases


def listed():
    return [
        # the smallest model: a step is a handful of microsecond kernels, so launches and their gaps are the cost
        dict(name="decode-tiny", kind="stack", dims="tiny", layers=1, batch=4, prompt=24, new=40, dtype="f16", act="silu", softcap=0.0),
        # one interactive user of the large model
        dict(name="decode-b1", kind="stack", dims="31b", layers=12, batch=1, prompt=48, new=48, dtype="bf16", act="silu", softcap=0.0),
        # the headline batch
        dict(name="decode-b32", kind="stack", dims="31b", layers=12, batch=32, prompt=64, new=64, dtype="bf16", act="silu", softcap=0.0),
        # a throughput-oriented batch, with the activation and the capped logits of the Gemma form
        dict(name="decode-b128", kind="stack", dims="31b", layers=12, batch=128, prompt=48, new=48, dtype="bf16", act="gelu", softcap=30.0),
        # a host executor driving one small layer call by call: the calls themselves are most of the cost
        dict(name="layer-tiny", kind="layer", dims="tiny", batch=4, ctx_lo=128, ctx_hi=128, is_global=True, dtype="f16", act="silu"),
        # the same on the large model with an odd batch of long, unequal contexts in a global layer
        dict(name="layer-31b-b19", kind="layer", dims="31b", batch=19, ctx_lo=300, ctx_hi=4000, is_global=True, dtype="bf16", act="silu"),
        # projections of a small decode batch (weight-bandwidth bound)
        dict(name="gemm-m8", kind="gemm", dims="31b", rows=8, dtype="f16"),
        # a ragged chunk of rows (neither bandwidth- nor tensor-bound by a wide margin)
        dict(name="gemm-m500", kind="gemm", dims="31b", rows=500, dtype="bf16"),
        # prefill-sized rows (tensor-bound)
        dict(name="gemm-m2048", kind="gemm", dims="31b", rows=2048, dtype="bf16"),
        # decode attention of 64 sequences, contexts 512..32768: sliding-window layers and global layers
        dict(name="attn-sliding-b64", kind="attn", heads=32, kv_heads=16, head_dim=128, batch=64, ctx_lo=512, ctx_hi=32768, window=1024, page=16, dtype="bf16"),
        dict(name="attn-global-b64", kind="attn", heads=32, kv_heads=16, head_dim=256, batch=64, ctx_lo=512, ctx_hi=32768, window=0, page=16, dtype="f16"),
        # the row kernels on a prefill chunk
        dict(name="rows-1000", kind="rows", dims="31b", rows=1000, dtype="bf16", act="silu"),
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["stack", "layer", "gemm", "gemm", "attn", "rows"])
    dtype = rng.choice(["f16", "bf16"])
    act = rng.choice(["silu", "gelu"])
    dims = rng.choice(["31b", "31b", "mid", "small", "tiny"])
    if kind == "stack":
        return dict(kind=kind, dims=dims, layers=rng.randint(1, 12), batch=_log_int(rng, 1, 128), prompt=rng.randint(8, 48),
                    new=rng.randint(8, 48), dtype=dtype, act=act, softcap=rng.choice([0.0, 30.0]))
    if kind == "layer":
        lo, hi = sorted((_log_int(rng, 16, 8192), _log_int(rng, 16, 8192)))
        return dict(kind=kind, dims=dims, batch=_log_int(rng, 1, 128), ctx_lo=lo, ctx_hi=hi, is_global=rng.random() < 0.5,
                    dtype=dtype, act=act)
    if kind == "gemm":
        return dict(kind=kind, dims=dims, rows=_log_int(rng, 1, 2048), dtype=dtype)
    if kind == "attn":
        heads, kv_heads = rng.choice([(32, 16), (32, 8), (64, 8), (8, 4)])
        hd = rng.choice([64, 128, 128, 256, 512])
        hi = _log_int(rng, 64, 32768)
        lo = _log_int(rng, 16, hi)
        most = max(1, min(64, 64 * 16 * 256 * 32768 // (kv_heads * hd * hi)))  # no more cache than the largest listed case
        return dict(kind=kind, heads=heads, kv_heads=kv_heads, head_dim=hd, batch=_log_int(rng, 1, most), ctx_lo=lo, ctx_hi=hi,
                    window=rng.choice([0, 0, 512, 1024]), page=rng.choice([16, 16, 32]), dtype=dtype)
    return dict(kind=kind, dims=dims, rows=_log_int(rng, 1, 4096), dtype=dtype, act=act)


# ---- inputs -----------------------------------------------------------------------------------------------------------
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _empty(*shape, dtype=torch.uint8):
    return torch.empty(shape, dtype=dtype, device="cuda")


def _quantise(x):
    s = (x.abs().amax(dim=1) / 448.0).clamp_min(1e-12)
    return (x / s[:, None]).to(torch.float8_e4m3fn).view(torch.uint8), s


def _fp8_rows(n, k, g, std=1.0):
    """[n, k] of N(0, std) as E4M3 bytes with a scale per row, drawn in pieces."""
    w, s = _empty(n, k), _empty(n, dtype=torch.float32)
    step = max(1, (16 << 20) // k)
    for r in range(0, n, step):
        m = min(step, n - r)
        w[r:r + m], s[r:r + m] = _quantise(torch.randn((m, k), generator=g, device="cuda") * std)
    return w, s


def _randn(shape, g, tdt):
    return torch.randn(shape, generator=g, device="cuda").to(tdt)


def _contexts(case):
    """The batch's context lengths: spread evenly over the case's range (the seed only shuffles them)."""
    lo, hi, b = case["ctx_lo"], case["ctx_hi"], case["batch"]
    return [hi if b == 1 else lo + (hi - lo) * i // (b - 1) for i in range(b)]


def _tables(case, contexts, window, page, g):
    """Block tables over shuffled physical pages.  Global: each sequence owns the pages of its context.  Sliding: a ring of
    pages that holds the window."""
    ring = window // page + 1
    need = [ring if window else -(-c // page) for c in contexts]
    width, total = max(need), sum(need)
    perm = torch.randperm(total, generator=g, device="cuda").to(torch.int32)
    tables = torch.zeros((len(need), width), dtype=torch.int32, device="cuda")
    at = 0
    for b, n in enumerate(need):
        tables[b, :n] = perm[at:at + n]
        at += n
    return tables, total


def _shuffled(contexts, seed):
    order = torch.randperm(len(contexts), generator=torch.Generator().manual_seed(seed)).tolist()
    return [contexts[i] for i in order]


def _rope_tables(n, half, tdt):
    inv = 10000.0 ** (-torch.arange(half, device="cuda", dtype=torch.float32) / half)
    ang = torch.arange(n, device="cuda", dtype=torch.float32)[:, None] * inv
    return ang.cos().to(tdt).contiguous(), ang.sin().to(tdt).contiguous()


# ---- stack ------------------------------------------------------------------------------------------------------------
def _stack_config(case):
    d = DIMS[case["dims"]]
    steps = case["prompt"] + case["new"]
    over = dict(num_layers=case["layers"], dtype=DTYPES[case["dtype"]][0], act=ACTS[case["act"]], logit_softcap=case["softcap"],
                prompt_len=case["prompt"], max_context=steps, max_steps=steps)
    if case["dims"] == "tiny":
        return stack.tiny_shape(case["batch"], **over)
    return stack.gemma31b_shape(case["batch"], hidden=d["hidden"], ffn=d["ffn"], vocab=d["vocab"], heads=d["heads"],
                                kv_heads=d["kv_heads"], sliding_head_dim=d["head_dim"], global_head_dim=d["global_head_dim"],
                                sliding_window=d["window"], **over)


def _prepare_stack(case, seed):
    """Random weights that decode as a trained model does: the residual branches scaled by 1 / sqrt(2 * layers), and an LM
    head tied to the embedding table (through a permutation of the tokens), so that the next token is a clear choice and
    not a tie among random logits."""
    cfg = _stack_config(case)
    g = _gen(seed)
    w = stack.random_weights(cfg, seed=seed)
    for layer in w.layers:
        layer["o_scale"] *= (2 * case["layers"]) ** -0.5
        layer["down_scale"] *= (2 * case["layers"]) ** -0.5
    emb, head, scale = w.head["embedding"], w.head["lm_head_w"], w.head["lm_head_scale"]
    perm = torch.randperm(cfg["vocab"], generator=g, device="cuda")
    step = max(1, (16 << 20) // cfg["hidden"])
    for r in range(0, cfg["vocab"], step):
        head[r:r + step], scale[r:r + step] = _quantise(emb[perm[r:r + step]].float() * 0.02)
    prompt = torch.randint(0, cfg["vocab"], (case["batch"], case["prompt"]), generator=g, device="cuda", dtype=torch.int32)
    return dict(kind="stack", stack=stack.DecodeStack(cfg, w), prompt=prompt.cpu().numpy(), steps=case["prompt"] + case["new"],
                tdt=DTYPES[case["dtype"]][1])


def _run_stack(s):
    st = s["stack"]
    st.reset(s["prompt"])
    st.run(s["steps"])
    tokens = st.tokens()
    hidden = torch.from_numpy(st.debug_read(0).view("int16")).view(s["tdt"])
    return {"tokens": tokens, "hidden": hidden}


# ---- layer ------------------------------------------------------------------------------------------------------------
def _layer_dims(case):
    d = dict(DIMS[case["dims"]])
    d["hd"] = d["global_head_dim"] if case["is_global"] else d["head_dim"]
    d["q"], d["kv"] = d["heads"] * d["hd"], d["kv_heads"] * d["hd"]
    return d


def _prepare_layer(case, seed):
    g, d, b = _gen(seed), _layer_dims(case), case["batch"]
    code, tdt = DTYPES[case["dtype"]]
    h, f, heads, kvh, hd = d["hidden"], d["ffn"], d["heads"], d["kv_heads"], d["hd"]
    window = 0 if case["is_global"] else d["window"]
    ctx = _shuffled(_contexts(case), seed)
    tables, blocks = _tables(case, ctx, window, PAGE, g)
    width = tables.shape[1]
    slots = blocks * PAGE
    k8, ks = _fp8_rows(slots * kvh, hd, g)
    v8, vs = _fp8_rows(slots * kvh, hd, g)
    ctx_t = torch.tensor(ctx, dtype=torch.int32, device="cuda")
    pos = ctx_t - 1
    page = ((pos // PAGE) % width).long()
    slot = tables.gather(1, page[:, None])[:, 0] * PAGE + pos % PAGE
    cos, sin = _rope_tables(max(ctx), hd // 2, tdt)
    params = PagedDecodeParams(b, heads, kvh, hd, PAGE, width, blocks, hd ** -0.5, window - 1 if window else -1)
    attn = PagedDecodeFp8Launcher(params)
    s = dict(kind="layer", d=d, act=ACTS[case["act"]], code=code, ctx=ctx_t, pos=pos, slot=slot.to(torch.int32), tables=tables,
             k8=k8, ks=ks, v8=v8, vs=vs, cos=cos, sin=sin, attn=attn, x=_randn((b, h), g, tdt),
             norm=launchers.FusedRmsnormFp8QuantLaunch(b, h, EPS), gamma1=_randn((h,), g, tdt) * 0.1 + 1, gamma2=_randn((h,), g, tdt) * 0.1 + 1,
             x8=_empty(b, h), xs=_empty(b, dtype=torch.float32), qkv=_empty(b, d["q"] + 2 * d["kv"], dtype=tdt),
             q8=_empty(b, d["q"]), qs=_empty(b, heads, dtype=torch.float32), a8=_empty(b, d["q"]), as_=_empty(b, dtype=torch.float32),
             attn_ws=_empty(max(256, attn.quant_workspace_bytes())), mid=_empty(b, h, dtype=tdt), out=_empty(b, h, dtype=tdt),
             h8=_empty(b, f), hs=_empty(b, dtype=torch.float32), work=_empty(gemm.gateup_workspace_bytes(b, f, h)))
    for name, n, k in (("qkv_w", d["q"] + 2 * d["kv"], h), ("o_w", h, d["q"]), ("gu_w", 2 * f, h), ("d_w", h, f)):
        s[name], s[name + "s"] = _fp8_rows(n, k, g, 0.02)
    return s


def _run_layer(s):
    d = s["d"]
    s["norm"].launch(s["x8"], s["xs"], s["x"], s["gamma1"])
    if not launchers.qkv_rope_fp8kv(s["x8"], s["qkv_w"], s["xs"], s["qkv_ws"], d["heads"], d["kv_heads"], d["hd"], s["cos"], s["sin"],
                                    s["pos"], s["slot"], s["q8"], s["qs"], s["k8"], s["v8"], s["ks"], s["vs"]):
        gemm.fp8_gemm_channelscale(s["qkv"], s["x8"], s["qkv_w"], s["xs"], s["qkv_ws"])
        launchers.rope_fp8kv(s["qkv"], d["heads"], d["kv_heads"], d["hd"], d["hd"], s["cos"], s["sin"], s["pos"], s["slot"],
                             s["q8"], s["qs"], s["k8"], s["v8"], s["ks"], s["vs"])
    s["attn"].launch_quant(s["q8"], s["k8"], s["v8"], s["a8"], s["as_"], s["code"], s["tables"], s["ctx"], s["attn_ws"],
                           k_scale_cache=s["ks"], v_scale_cache=s["vs"], q_scale_cache=s["qs"])
    gemm.fp8_gemm_channelscale(s["mid"], s["a8"], s["o_w"], s["as_"], s["o_ws"], residual=s["x"])
    s["norm"].launch(s["x8"], s["xs"], s["mid"], s["gamma2"])
    gemm.fp8_gemm_gateup_act_quant(s["h8"], s["hs"], s["x8"], s["gu_w"], s["xs"], s["gu_ws"], s["act"], s["code"], s["work"])
    gemm.fp8_gemm_channelscale(s["out"], s["h8"], s["d_w"], s["hs"], s["d_ws"], residual=s["mid"])
    return {"out": s["out"], "mid": s["mid"], "q_scale": s["qs"], "attn_scale": s["as_"], "h_scale": s["hs"]}


# ---- gemm -------------------------------------------------------------------------------------------------------------
def _projections(case):
    d = DIMS[case["dims"]]
    q, kv = d["heads"] * d["head_dim"], d["kv_heads"] * d["head_dim"]
    return [("qkv", q + 2 * kv, d["hidden"], False), ("o", d["hidden"], q, True), ("gateup", 2 * d["ffn"], d["hidden"], False),
            ("down", d["hidden"], d["ffn"], True)]


def _prepare_gemm(case, seed):
    g, m, tdt = _gen(seed), case["rows"], DTYPES[case["dtype"]][1]
    ops = []
    for _, n, k, residual in _projections(case):
        a8, asc = _fp8_rows(m, k, g)
        w8, wsc = _fp8_rows(n, k, g, 0.02)
        ops.append((_empty(m, n, dtype=tdt), a8, w8, asc, wsc, _randn((m, n), g, tdt) if residual else None))
    return dict(kind="gemm", ops=ops)


def _run_gemm(s):
    for out, a8, w8, asc, wsc, residual in s["ops"]:
        gemm.fp8_gemm_channelscale(out, a8, w8, asc, wsc, residual=residual)
    return [op[0] for op in s["ops"]]


# ---- attn -------------------------------------------------------------------------------------------------------------
def _prepare_attn(case, seed):
    g, b, hd, kvh, page = _gen(seed), case["batch"], case["head_dim"], case["kv_heads"], case["page"]
    ctx = _shuffled(_contexts(case), seed)
    tables, blocks = _tables(case, ctx, case["window"], page, g)
    k8, ks = _fp8_rows(blocks * page * kvh, hd, g)
    v8, vs = _fp8_rows(blocks * page * kvh, hd, g)
    q8, qs = _fp8_rows(b * case["heads"], hd, g)
    attn = PagedDecodeFp8Launcher(PagedDecodeParams(b, case["heads"], kvh, hd, page, tables.shape[1], blocks, hd ** -0.5,
                                                    case["window"] - 1 if case["window"] else -1))
    return dict(kind="attn", attn=attn, q8=q8, qs=qs, k8=k8, ks=ks, v8=v8, vs=vs, tables=tables,
                ctx=torch.tensor(ctx, dtype=torch.int32, device="cuda"), ws=_empty(max(256, attn.params.workspace_bytes())),
                out=_empty(b, case["heads"], hd, dtype=DTYPES[case["dtype"]][1]))


def _run_attn(s):
    s["attn"].launch(s["q8"], s["k8"], s["v8"], s["out"], s["tables"], s["ctx"], workspace=s["ws"], k_scale_cache=s["ks"],
                     v_scale_cache=s["vs"], q_scale_cache=s["qs"])
    return s["out"]


# ---- rows -------------------------------------------------------------------------------------------------------------
def _prepare_rows(case, seed):
    g, t, d = _gen(seed), case["rows"], DIMS[case["dims"]]
    tdt = DTYPES[case["dtype"]][1]
    h, f, v, heads, kvh, hd = d["hidden"], d["ffn"], d["vocab"], d["heads"], d["kv_heads"], d["head_dim"]
    q, kv = heads * hd, kvh * hd
    cos, sin = _rope_tables(t, hd // 2, tdt)
    f32 = torch.float32
    n = min(t, ARGMAX_ROWS)
    return dict(kind="rows", d=d, x=_randn((t, h), g, tdt), res=_randn((t, h), g, tdt), gamma=_randn((h,), g, tdt) * 0.1 + 1,
                a=_randn((t, q), g, tdt), gu=_randn((t, 2 * f), g, tdt), qkv=_randn((t, q + 2 * kv), g, tdt), cos=cos, sin=sin,
                pos=torch.arange(t, dtype=torch.int32, device="cuda"),
                slot=torch.randperm(t, generator=g, device="cuda").to(torch.int32), logits=_randn((n, v), g, f32),
                add_norm=launchers.FusedAddRmsnormFp8QuantLaunch(t, h, EPS), quant=launchers.QuantizeFp8PerTokenLaunch(t, q),
                act=launchers.FusedActMulFp8QuantLaunch(t, f, ACTS[case["act"]]), argmax=launchers.ArgmaxLaunch(n, v),
                res_out=_empty(t, h, dtype=tdt), x8=_empty(t, h), xs=_empty(t, dtype=f32), a8=_empty(t, q), as_=_empty(t, dtype=f32),
                h8=_empty(t, f), hs=_empty(t, dtype=f32), q8=_empty(t, q), qs=_empty(t, heads, dtype=f32), k8=_empty(t, kv),
                v8=_empty(t, kv), ks=_empty(t * kvh, dtype=f32), vs=_empty(t * kvh, dtype=f32), tok=_empty(n, dtype=torch.int32))


def _run_rows(s):
    d = s["d"]
    s["add_norm"].launch(s["x8"], s["xs"], s["res_out"], s["x"], s["res"], s["gamma"])
    launchers.rope_fp8kv(s["qkv"], d["heads"], d["kv_heads"], d["head_dim"], d["head_dim"], s["cos"], s["sin"], s["pos"], s["slot"],
                         s["q8"], s["qs"], s["k8"], s["v8"], s["ks"], s["vs"])
    s["quant"].launch(s["a8"], s["as_"], s["a"])
    s["act"].launch(s["h8"], s["hs"], s["gu"])
    s["argmax"].launch(s["logits"], s["tok"])
    return {k: s[k] for k in ("res_out", "x8", "xs", "q8", "qs", "k8", "v8", "ks", "vs", "a8", "as_", "h8", "hs", "tok")}


# ---- the interface ----------------------------------------------------------------------------------------------------
def prepare(case, seed):
    return {"stack": _prepare_stack, "layer": _prepare_layer, "gemm": _prepare_gemm, "attn": _prepare_attn,
            "rows": _prepare_rows}[case["kind"]](case, seed)


def run(state):
    return {"stack": _run_stack, "layer": _run_layer, "gemm": _run_gemm, "attn": _run_attn, "rows": _run_rows}[state["kind"]](state)


def _attn_work(batch, heads, kv_heads, hd, contexts, out_bytes):
    tokens = sum(contexts)
    return (tokens * kv_heads * (2 * hd + 8) + batch * heads * (hd * (1 + out_bytes) + 4) + 4 * batch, 4.0 * tokens * heads * hd)


def _layer_work(d, hd, m, contexts):
    """One layer on m tokens whose contexts (tokens attended) are given: weights once, residual in and out, KV read and written."""
    h, f, q, kv = d["hidden"], d["ffn"], d["heads"] * hd, d["kv_heads"] * hd
    params = (q + 2 * kv) * h + h * q + 3 * f * h
    by, fl = _attn_work(m, d["heads"], d["kv_heads"], hd, contexts, 0)
    return params + 4 * (q + 2 * kv + 2 * f + 2 * h) + 4 * h + 4 * m * h + m * d["kv_heads"] * (2 * hd + 8) + by, 2.0 * m * params + fl


def work(case):
    kind = case["kind"]
    if kind == "attn":
        ctx = [min(c, case["window"]) if case["window"] else c for c in _contexts(case)]
        by, fl = _attn_work(case["batch"], case["heads"], case["kv_heads"], case["head_dim"], ctx, 2)
        return {"bytes": by, "flops": fl}
    d = DIMS[case["dims"]]
    if kind == "gemm":
        m = case["rows"]
        ops = _projections(case)
        return {"bytes": sum(n * k + m * k + 2 * m * n * (2 if r else 1) + 4 * (m + n) for _, n, k, r in ops),
                "flops": sum(2.0 * m * n * k for _, n, k, _ in ops)}
    if kind == "rows":
        t, h, f = case["rows"], d["hidden"], d["ffn"]
        q, kv = d["heads"] * d["head_dim"], d["kv_heads"] * d["head_dim"]
        qkv = q + 2 * kv
        return {"bytes": t * (h * 7 + 3 * qkv + 3 * q + 5 * f) + 2 * t * d["head_dim"] + 4 * min(t, ARGMAX_ROWS) * d["vocab"],
                "flops": 8.0 * t * (h + q + qkv + 3 * f)}
    if kind == "layer":
        g = _layer_dims(case)
        ctx = [c if case["is_global"] else min(c, g["window"]) for c in _contexts(case)]
        by, fl = _layer_work(g, g["hd"], case["batch"], ctx)
        return {"bytes": by, "flops": fl}
    cfg = _stack_config(case)
    b, steps = case["batch"], case["prompt"] + case["new"]
    by = fl = 0.0
    for layer in range(case["layers"]):
        is_global = cfg["global_every"] and (layer + 1) % cfg["global_every"] == 0
        hd = cfg["global_head_dim"] if is_global else cfg["sliding_head_dim"]
        for step in range(steps):
            x, y = _layer_work(d, hd, b, [step + 1 if is_global else min(step + 1, cfg["sliding_window"])] * b)
            by, fl = by + x - 4 * b * d["hidden"], fl + y  # (inside a stack the residual need not leave the chip)
    params = d["vocab"] * d["hidden"]
    return {"bytes": by + steps * (params + 4 * d["vocab"] + 2 * b * d["hidden"]), "flops": fl + steps * 2.0 * b * params}


def tolerance(case):
    kind = case["kind"]
    if kind == "rows":  # one rounding of a row's f32 sum or maximum; bytes that lie on a rounding boundary of the new scale
        return {"rel": 2e-6, "max": 1e-2, "differ": 2e-3}
    if kind == "gemm":  # f32 sums in another order, rounded to 16 bits
        return {"rel": 2e-3, "max": 2e-2}
    if kind == "attn":  # f32 softmax in another order, probabilities at 16 bits
        return {"rel": 4e-3, "max": 5e-2}
    # whole layers and stacks: a 16-bit rounding that falls the other way moves an FP8 code of the next stage
    return {"rel": 1e-2, "max": 0.3, "differ": 1e-2}
