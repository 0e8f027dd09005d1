"""Performance cases: what a user of the library has it do, through its public entry points, from the smallest call to the largest.

Two families of work are here, as the library serves them:

* the quantised Llama-style models over the `qserve_backend` operators -- one linear layer, decode attention over the paged INT4 / INT8 cache,
  a prompt's attention block and feed-forward block in the operator order of the reference model code, and whole decoder layers of a decode
  step, replayed as a CUDA graph with the fused operators (what `qserve_b200.decode.DecodeRunner` does for a whole model);
* the unquantised hybrid decoders (`qserve_b200.hybrid.HybridDecoder`): a layer of differential attention, of the gated delta rule and of the
  state space recurrence over a step of prompts, and a whole decode step with its logits.

Sizes are those of `qserve_b200.modelcfg.MODELS` (Llama-3-8B, Mistral-7B, Llama-2-7B) and of `bench.py`'s hybrid stacks (width 2048: 16 heads,
4 key/value heads of 128, feed-forward 8192).  All inputs are random and made from the seed alone.
"""
import math

import torch

F64 = torch.float64
HALF, BF16, F32 = torch.float16, torch.bfloat16, torch.float32
PAGE = 64  # tokens of a cache page
D = 128    # head size

# hidden, feed-forward, query heads, key/value heads, rotary base, norm eps
LLAMA = {
    "llama-3-8b": (4096, 14336, 32, 8, 500000.0, 1e-5),
    "mistral-7b": (4096, 14336, 32, 8, 10000.0, 1e-5),
    "llama-2-7b": (4096, 11008, 32, 32, 10000.0, 1e-5),
}


def listed():
    return [
        # the smallest call: one 4096 x 4096 linear layer (an output projection) for 16 tokens
        {"name": "linear_w4_m16", "kind": "linear", "mode": "chn", "m": 16, "n": 4096, "k": 4096},
        # the widest linear layer for a step that mixes a short prompt with decoded tokens
        {"name": "linear_w4_g128_m250", "kind": "linear", "mode": "grp", "m": 250, "n": 28672, "k": 4096},
        # decode attention of Llama-3-8B at batch 64, contexts of up to 1024 tokens, INT4 cache
        {"name": "attention_kv4_b64", "kind": "decode_attention", "model": "llama-3-8b", "bits": 4, "batch": 64, "ctx": 1024},
        # few long contexts over the INT8 cache
        {"name": "attention_kv8_long", "kind": "decode_attention", "model": "mistral-7b", "bits": 8, "batch": 4, "ctx": 8000},
        # a prompt step's attention block: qkv projection, rotary + cache append, causal attention, output projection
        {"name": "prompt_attention", "kind": "prompt_attention", "model": "llama-3-8b", "mode": "chn", "bits": 4, "prompts": 8, "ctx": 1024},
        # a prompt step's feed-forward block with grouped INT4 weights
        {"name": "prompt_mlp_g128", "kind": "prompt_mlp", "model": "llama-3-8b", "mode": "grp", "m": 5000},
        # one decoder layer of the headline decode step
        {"name": "decode_layer_w4kv4_b64", "kind": "decode_layer", "model": "llama-3-8b", "mode": "chn", "bits": 4, "batch": 64, "ctx": 1024},
        # the 8-bit path at a larger batch
        {"name": "decode_layer_w8kv8_b128", "kind": "decode_layer", "model": "mistral-7b", "mode": "w8", "bits": 8, "batch": 128, "ctx": 1024},
        # hybrid decoders: one layer each over a step of prompts, and a decode step of a small stack
        {"name": "hybrid_attention_prompt", "kind": "hybrid_attention", "width": 2048, "prompts": 4, "ctx": 2048},
        {"name": "hybrid_delta_prompt", "kind": "hybrid_delta", "width": 2048, "prompts": 4, "ctx": 2048},
        {"name": "hybrid_state_space_prompt", "kind": "hybrid_state_space", "width": 2048, "prompts": 4, "ctx": 2048},
        {"name": "hybrid_decode_b64", "kind": "hybrid_decode", "width": 2048, "batch": 64, "ctx": 1024},
    ]


def draw(rng):
    def log(lo, hi):
        return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))

    kind = rng.choice(["linear", "linear", "decode_attention", "decode_attention", "prompt_attention", "prompt_mlp", "decode_layer", "decode_layer",
                       "hybrid_attention", "hybrid_delta", "hybrid_state_space", "hybrid_decode"])
    model = rng.choice(sorted(LLAMA))
    H, I, hq, hkv = LLAMA[model][:4]
    mode, bits = rng.choice(["chn", "grp", "w8"]), rng.choice([4, 8])
    if kind == "linear":
        n, k = rng.choice([((hq + 2 * hkv) * D, H), (H, H), (2 * I, H), (H, I)])
        return {"kind": kind, "mode": mode, "m": log(1, 2000), "n": n, "k": k}
    if kind == "decode_attention":
        batch = log(1, 128)
        return {"kind": kind, "model": model, "bits": bits, "batch": batch, "ctx": log(32, min(8000, 65536 // batch))}
    if kind == "prompt_attention":
        return {"kind": kind, "model": model, "mode": mode, "bits": bits, "prompts": rng.randint(1, 8), "ctx": log(16, 1024)}
    if kind == "prompt_mlp":
        return {"kind": kind, "model": model, "mode": mode, "m": log(16, 5000)}
    if kind == "decode_layer":
        return {"kind": kind, "model": model, "mode": mode, "bits": bits, "batch": log(1, 128), "ctx": log(32, 1024)}
    if kind == "hybrid_decode":
        return {"kind": kind, "width": rng.choice([1024, 2048]), "batch": log(1, 64), "ctx": log(32, 1024)}
    return {"kind": kind, "width": rng.choice([1024, 2048]), "prompts": rng.randint(1, 4), "ctx": log(64, 2048)}


# ------------------------------------------------------------------------------------------------------------------------
# what both `prepare` and `exact` make from the seed
# ------------------------------------------------------------------------------------------------------------------------
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _normal(g, *shape, s=1.0, dtype=F32):
    return (torch.randn(*shape, device="cuda", generator=g) * s).to(dtype)


def _uniform(g, lo, hi, *shape):
    return torch.rand(*shape, device="cuda", generator=g) * (hi - lo) + lo


def _ints(g, lo, hi, shape, dtype):
    return torch.randint(lo, hi, shape, dtype=dtype, device="cuda", generator=g)


def _lengths(count, ctx):
    """Ragged lengths from about half of `ctx` up to `ctx`, the same for every seed."""
    return [ctx - (i * 7919) % max(1, ctx // 2) for i in range(count)]


def _linear(g, n, k, mode):
    """Weights of a quantised linear layer in the buffers the operators take; outputs of unit-variance inputs come out around one."""
    target = k ** -0.5
    if mode == "w8":
        return {"mode": mode, "w": _ints(g, -127, 128, (n, k), torch.int8), "s": (_uniform(g, 0.8, 1.2, n) * target / 73.0).half()}
    w = {"mode": mode, "w": _ints(g, -128, 128, (n, k // 2), torch.int8)}
    if mode == "chn":
        w["s"] = (_uniform(g, 0.8, 1.2, n) * target / 4.6).half()
        w["sz"] = (_ints(g, 7, 9, (n,), torch.int32).float() * w["s"].float()).half()
        return w
    s2, z = _ints(g, 1, 9, (k // 128, n), torch.int32), _ints(g, 7, 9, (k // 128, n), torch.int32)
    w["s2"], w["z2"] = s2.to(torch.int8), (-z * s2).to(torch.int8)
    w["s"] = (_uniform(g, 0.8, 1.2, n) * target / (4.6 * 4.5)).half()
    return w


def _codes(g, m, k):
    """An INT8 activation as the per-token quantisation leaves it: codes, scale, and the sum of the row."""
    x = _normal(g, m, k)
    amax = x.abs().amax(1)
    q = torch.round(x * (127.0 / amax)[:, None]).to(torch.int8)
    scale = (amax / 127.0).half()
    return q, scale, (q.float().sum(1) * scale.float()).half()


def _pools(g, lens, hkv, bits):
    """K and V pools of one layer with random contents, their address table and the page table: page = codes [hkv][64][D * bits / 8], scales and
    zeros [hkv][64] fp16."""
    blocks = (max(lens) + PAGE - 1) // PAGE
    n = len(lens) * blocks
    code = hkv * PAGE * D * bits // 8
    pools = []
    for _ in range(2):
        p = _ints(g, 0, 256, (n, code + hkv * PAGE * 4), torch.uint8)
        meta = p[:, code:].view(HALF).view(n, 2, hkv, PAGE)
        top = 2 ** bits - 1
        meta[:, 0] = _uniform(g, 1.0, 4.0, n, hkv, PAGE).half() / top
        meta[:, 1] = _uniform(g, 0.3 * top, 0.7 * top, n, hkv, PAGE).half()
        pools.append(p)
    pages = torch.randperm(n, device="cuda", generator=g).view(len(lens), blocks)
    table = torch.stack([p.data_ptr() + pages * p.shape[1] for p in pools], 1).contiguous()
    return pools, pages, table


def _llama_weights(g, case):
    H, I, hq, hkv = LLAMA[case["model"]][:4]
    mode = case["mode"]
    return {"qkv": _linear(g, (hq + 2 * hkv) * D, H, mode), "o": _linear(g, H, hq * D, mode), "gate_up": _linear(g, 2 * I, H, mode),
            "down": _linear(g, H, I, mode)}


def _hybrid_sizes(width):
    return width, width // 128, max(1, width // 512)  # width, heads, key/value heads


def _attention_weights(g, W, H, G, p):
    r = lambda *s, sc: _normal(g, *s, s=sc, dtype=BF16)
    w = {p + "q": r(H * 2 * D, W, sc=W ** -0.5), p + "k": r(G * 2 * D, W, sc=W ** -0.5), p + "v": r(G * D, W, sc=W ** -0.5)}
    for n in ("lq1", "lk1", "lq2", "lk2"):
        w[p + n] = r(D, sc=0.1)
    w[p + "o"] = r(W, H * D, sc=(H * D) ** -0.5)
    return w


def _delta_weights(g, W, H, G, p):
    r = lambda *s, sc: _normal(g, *s, s=sc, dtype=BF16)
    w = {}
    for n, c in (("q", G * D), ("k", G * D), ("v", H * D)):
        w[p + n], w[p + n + ".conv"] = r(c, W, sc=W ** -0.5), r(c, 4, sc=0.5)
    w[p + "b"], w[p + "a"], w[p + "g"] = r(H, W, sc=W ** -0.5), r(H, W, sc=W ** -0.5), r(H * D, W, sc=W ** -0.5)
    w[p + "A_log"], w[p + "dt_bias"], w[p + "norm"] = r(H, sc=0.5), r(H, sc=0.5), 1.0 + r(D, sc=0.1)
    w[p + "o"] = r(W, H * D, sc=(H * D) ** -0.5)
    return w


SSM_STATE, SSM_DIM, SSM_GROUPS, SSM_CONV = 128, 64, 8, 4


def _state_space_weights(g, W, p):
    r = lambda *s, sc: _normal(g, *s, s=sc, dtype=BF16)
    H = 2 * W // SSM_DIM
    inner, ch = 2 * W, 2 * W + 2 * SSM_GROUPS * SSM_STATE
    return {p + "in": r(inner + ch + H, W, sc=W ** -0.5), p + "conv": r(ch, SSM_CONV, sc=0.5), p + "conv.b": r(ch, sc=0.1),
            p + "dt_bias": r(H, sc=0.5) - 2.0, p + "A_log": r(H, sc=0.5), p + "D": 1.0 + r(H, sc=0.1), p + "norm": 1.0 + r(inner, sc=0.1),
            p + "o": r(W, inner, sc=inner ** -0.5)}


HYBRID_VOCAB, BUCKETS, MUL_PREV, MUL_CUR, HYBRID_FF, EPS = 4096, 4093, 131, 11, 4, 1e-5


def _hybrid_weights(g, case):
    W, H, G = _hybrid_sizes(case["width"])
    r = lambda *s, sc: _normal(g, *s, s=sc, dtype=BF16)
    if case["kind"] == "hybrid_state_space":
        return {"embed": r(HYBRID_VOCAB, W, sc=W ** -0.5), "final.norm": 1.0 + r(W, sc=0.1), "l0.norm1": 1.0 + r(W, sc=0.1),
                **_state_space_weights(g, W, "l0.mix.")}
    w = {"embed": r(HYBRID_VOCAB, W, sc=1.0), "head": r(HYBRID_VOCAB, W, sc=W ** -0.5), "final.norm": r(W, sc=0.1),
         "bigram": r(BUCKETS + 1, W, sc=0.5), "l0.norm1": r(W, sc=0.1)}
    if case["kind"] != "hybrid_delta":
        w.update(_attention_weights(g, W, H, G, "l0.mix."))
    if case["kind"] == "hybrid_delta":
        w.update(_delta_weights(g, W, H, G, "l0.mix."))
    if case["kind"] == "hybrid_decode":
        w["l1.norm1"] = r(W, sc=0.1)
        w.update(_delta_weights(g, W, H, G, "l1.mix."))
        for p in ("l0.", "l1."):
            ff = HYBRID_FF * W
            w[p + "norm2"], w[p + "mlp.gate"], w[p + "mlp.up"] = r(W, sc=0.1), r(ff, W, sc=W ** -0.5), r(ff, W, sc=W ** -0.5)
            w[p + "mlp.down"] = r(W, ff, sc=ff ** -0.5)
    return w


def _hybrid_lens(case):
    return _lengths(case["prompts"], case["ctx"])


def _decode_cache(g, case, runs):
    """Contents of the caches of a decode step: keys and values of every position, recurrent state and convolution inputs of every slot."""
    _, kv = runs[0], runs[1]
    for t in (runs[0]["k"], runs[0]["v"]):
        t.copy_(_normal(g, *t.shape, dtype=BF16))
    kv["state"].copy_(_normal(g, *kv["state"].shape, s=0.1))
    kv["conv"].copy_(_normal(g, *kv["conv"].shape))


# ------------------------------------------------------------------------------------------------------------------------
# prepare / run
# ------------------------------------------------------------------------------------------------------------------------
def _apply(lin, xq, scale, asum, out):
    import qserve_backend.qgemm_w4a8_per_chn as chn
    import qserve_backend.qgemm_w4a8_per_group as grp
    import qserve_backend.qgemm_w8a8 as w8

    if lin["mode"] == "chn":
        chn.gemm_forward_cuda(xq, lin["w"], lin["s"], scale, lin["sz"], asum, out)
    elif lin["mode"] == "grp":
        grp.gemm_forward_cuda(xq, lin["w"], lin["z2"], lin["s2"], lin["s"], scale, out)
    else:
        w8.w8a8_gemm_forward_cuda(xq, lin["w"], lin["s"], scale, out)


def _rms_quant(mode, q, x, gamma, asum, scale, eps):
    import qserve_backend.layernorm_ops as ln

    if mode == "chn":
        ln.rms_norm_general_fuse_sum(q, x, gamma, asum, scale, eps, True)
    else:
        ln.rms_norm_general(q, x, gamma, scale, eps, True)


def _quant(mode, q, x, asum, scale):
    import qserve_backend.fused_kernels as fk

    if mode == "chn":
        fk.invoke_quant_fuse_sum(q, x, asum, scale)
    else:
        fk.invoke_quant(q, x, scale)


def _prepare_linear(case, seed):
    g = _gen(seed)
    lin = _linear(g, case["n"], case["k"], case["mode"])
    xq, scale, asum = _codes(g, case["m"], case["k"])
    return {"lin": lin, "x": xq, "scale": scale, "sum": asum, "out": torch.empty(case["m"], case["n"], dtype=HALF, device="cuda")}


def _run_linear(case, s):
    _apply(s["lin"], s["x"], s["scale"], s["sum"], s["out"])
    return s["out"]


def _prepare_decode_attention(case, seed):
    g = _gen(seed)
    _, _, hq, hkv, base, _ = LLAMA[case["model"]]
    lens = [n + 1 for n in _lengths(case["batch"], case["ctx"])]  # the new token included
    pools, pages, table = _pools(g, lens, hkv, case["bits"])
    B = case["batch"]
    qkv = _normal(g, B, (hq + 2 * hkv) * D, dtype=HALF)
    return {"pools": pools, "pages": pages, "table": table, "qkv": qkv, "lens": torch.tensor(lens, dtype=torch.int32, device="cuda"), "top": max(lens),
            "hq": hq, "hkv": hkv, "base": base, "spt": hkv * D * case["bits"] // 8}


def _run_decode_attention(case, s):
    import qserve_backend.fused_attention as fa

    hq, hkv = s["hq"], s["hkv"]
    q, k, v = s["qkv"].split([hq * D, hkv * D, hkv * D], dim=-1)
    out = fa.single_query_attention(q.reshape(-1, hq, D), k.reshape(-1, hkv, D), v.reshape(-1, hkv, D), s["table"], s["lens"], None, 8192, PAGE, s["spt"],
                                    s["top"], D, s["base"], True, case["bits"] == 4, True)
    return {"out": out, "k": s["pools"][0], "v": s["pools"][1]}


def _prepare_prompt_attention(case, seed):
    g = _gen(seed)
    H, _, hq, hkv, base, eps = LLAMA[case["model"]]
    lens = _lengths(case["prompts"], case["ctx"])
    T = sum(lens)
    xq, scale, asum = _codes(g, T, H)
    pools, pages, table = _pools(g, lens, hkv, case["bits"])
    lin = {"qkv": _linear(g, (hq + 2 * hkv) * D, H, case["mode"]), "o": _linear(g, H, hq * D, case["mode"])}
    cu = torch.tensor([0] + lens, dtype=torch.int32, device="cuda").cumsum(0).to(torch.int32)
    e = lambda *sh, dt=HALF: torch.empty(*sh, dtype=dt, device="cuda")
    return {"x": xq, "scale": scale, "sum": asum, "pools": pools, "pages": pages, "table": table, "lin": lin, "cu": cu, "top": max(lens), "T": T,
            "lens": torch.tensor(lens, dtype=torch.int32, device="cuda"), "qkv": e(T, (hq + 2 * hkv) * D), "aq": e(T, hq * D, dt=torch.int8),
            "ascale": e(T), "asum": e(T), "out": e(T, H), "hq": hq, "hkv": hkv, "base": base, "spt": hkv * D * case["bits"] // 8}


def _run_prompt_attention(case, s):
    import qserve_backend.fused_attention as fa
    from qserve_b200.backend import flash_attn_varlen_func

    hq, hkv, T = s["hq"], s["hkv"], s["T"]
    _apply(s["lin"]["qkv"], s["x"], s["scale"], s["sum"], s["qkv"])
    pad = fa.compute_padding_offsets(s["cu"], s["top"], T)
    fa.apply_bias_rope_update_kv_cache(s["qkv"], s["lens"], pad, s["table"], hq, hkv, s["top"], PAGE, s["spt"], D, s["base"], 8192, True,
                                       case["bits"] == 4, True)
    q, k, v = s["qkv"].split([hq * D, hkv * D, hkv * D], dim=-1)
    a = flash_attn_varlen_func(q.view(T, hq, D), k.view(T, hkv, D), v.view(T, hkv, D), s["cu"], s["cu"], s["top"], s["top"], 0.0, None, True)
    _quant(case["mode"], s["aq"], a.view(T, hq * D), s["asum"], s["ascale"])
    _apply(s["lin"]["o"], s["aq"], s["ascale"], s["asum"], s["out"])
    return {"out": s["out"], "attention": a, "qkv": s["qkv"], "k": s["pools"][0], "v": s["pools"][1]}


def _prepare_prompt_mlp(case, seed):
    g = _gen(seed)
    H, I, _, _, _, eps = LLAMA[case["model"]]
    m = case["m"]
    e = lambda *sh, dt=HALF: torch.empty(*sh, dtype=dt, device="cuda")
    return {"x": _normal(g, m, H, dtype=HALF), "gamma": (1.0 + _normal(g, H, s=0.1)).half(), "gate_up": _linear(g, 2 * I, H, case["mode"]),
            "down": _linear(g, H, I, case["mode"]), "q": e(m, H, dt=torch.int8), "scale": e(m), "sum": e(m), "gu": e(m, 2 * I), "act": e(m, I),
            "aq": e(m, I, dt=torch.int8), "out": e(m, H), "eps": eps}


def _run_prompt_mlp(case, s):
    import qserve_backend.activation_ops as act

    _rms_quant(case["mode"], s["q"], s["x"], s["gamma"], s["sum"], s["scale"], s["eps"])
    _apply(s["gate_up"], s["q"], s["scale"], s["sum"], s["gu"])
    act.silu_and_mul(s["act"], s["gu"])
    _quant(case["mode"], s["aq"], s["act"], s["sum"], s["scale"])
    _apply(s["down"], s["aq"], s["scale"], s["sum"], s["out"])
    return {"out": s["x"] + s["out"], "act": s["act"], "codes": s["q"]}


def _layer(case, s):
    """One decoder layer of a decode step, in the order of `DecodeRunner`'s fused path; leaves the new hidden rows in s["y"]."""
    from qserve_b200 import backend as ext

    w, chn = s["w"], case["mode"] == "chn"
    hq, hkv, asum = s["hq"], s["hkv"], s["sum"] if chn else None
    _rms_quant(case["mode"], s["q"], s["x"], s["gamma"][0], s["sum"], s["scale"], s["eps"])
    _apply(w["qkv"], s["q"], s["scale"], s["sum"], s["qkv"])
    q, k, v = s["qkv"].split([hq * D, hkv * D, hkv * D], dim=-1)
    ext.single_query_attention_quant(q.reshape(-1, hq, D), k.reshape(-1, hkv, D), v.reshape(-1, hkv, D), s["table"], s["lens"], 8192, PAGE, s["spt"],
                                     s["top"], D, s["base"], case["bits"] == 4, True, s["aq"], s["scale"], asum)
    _apply(w["o"], s["aq"], s["scale"], s["sum"], s["o"])
    ext.add_rms_norm_general(s["q"], s["h"], s["x"], s["o"], s["gamma"][1], asum, s["scale"], s["eps"])
    _apply(w["gate_up"], s["q"], s["scale"], s["sum"], s["gu"])
    ext.silu_and_mul_quant(s["mq"], s["gu"], asum, s["scale"])
    _apply(w["down"], s["mq"], s["scale"], s["sum"], s["o"])
    torch.add(s["h"], s["o"], out=s["y"])


def _prepare_decode_layer(case, seed):
    g = _gen(seed)
    H, I, hq, hkv, base, eps = LLAMA[case["model"]]
    B = case["batch"]
    lens = [n + 1 for n in _lengths(B, case["ctx"])]
    e = lambda *sh, dt=HALF: torch.empty(*sh, dtype=dt, device="cuda")
    s = {"x": _normal(g, B, H, dtype=HALF), "gamma": [(1.0 + _normal(g, H, s=0.1)).half() for _ in range(2)], "w": _llama_weights(g, case)}
    s["pools"], s["pages"], s["table"] = _pools(g, lens, hkv, case["bits"])
    s.update(lens=torch.tensor(lens, dtype=torch.int32, device="cuda"), top=max(lens), hq=hq, hkv=hkv, base=base, eps=eps, spt=hkv * D * case["bits"] // 8,
             q=e(B, H, dt=torch.int8), aq=e(B, hq * D, dt=torch.int8), mq=e(B, I, dt=torch.int8), scale=e(B), sum=e(B), qkv=e(B, (hq + 2 * hkv) * D),
             o=e(B, H), h=e(B, H), gu=e(B, 2 * I), y=e(B, H))
    _layer(case, s)  # eager once: work spaces and kernel attributes
    torch.cuda.synchronize()
    s["graph"] = torch.cuda.CUDAGraph()
    with torch.cuda.graph(s["graph"]):
        _layer(case, s)
    return s


def _run_decode_layer(case, s):
    s["graph"].replay()
    return {"hidden": s["y"], "middle": s["h"], "qkv": s["qkv"], "k": s["pools"][0], "v": s["pools"][1]}


def _rotary():
    from qserve_b200.modelcfg import RotaryConfig

    return RotaryConfig(D // 2, 1e6, 4.0, 4096, 32.0, 1.0)


def _hybrid_model(case, w):
    from qserve_b200.hybrid import HybridDecoder
    from qserve_b200.modelcfg import AttentionMixerConfig, DeltaMixerConfig, HybridConfig, HybridLayerConfig, MlpConfig, StateSpaceMixerConfig

    W, H, G = _hybrid_sizes(case["width"])
    if case["kind"] == "hybrid_state_space":
        mix = StateSpaceMixerConfig(2 * W // SSM_DIM, SSM_STATE, SSM_DIM, SSM_GROUPS, SSM_CONV, SSM_GROUPS)
        cfg = HybridConfig("Tumitar", HYBRID_VOCAB, W, EPS, (HybridLayerConfig("state_space", mix, None),), norm_offset=0.0, block="sequential",
                           embed_scale=8.0, tied_head=True)
        return HybridDecoder(cfg, w, BF16, torch.device("cuda", torch.cuda.current_device()))
    att = HybridLayerConfig("attention", AttentionMixerConfig(H, G, D, D, _rotary(), D ** -0.5, maps=2, diff=0.5, head_norm=True), None)
    dlt = HybridLayerConfig("delta", DeltaMixerConfig(H, G, D, D, 4), None)
    layers = {"hybrid_attention": (att,), "hybrid_delta": (dlt,)}.get(case["kind"])
    if layers is None:
        ff = MlpConfig("dense", HYBRID_FF * W)
        layers = (HybridLayerConfig("attention", att.mixer, ff), HybridLayerConfig("delta", dlt.mixer, ff))
    cfg = HybridConfig("Rizurax", HYBRID_VOCAB, W, EPS, layers, pair_buckets=BUCKETS, pair_mul_prev=MUL_PREV, pair_mul_cur=MUL_CUR)
    return HybridDecoder(cfg, w, BF16, torch.device("cuda", torch.cuda.current_device()))


def _hybrid_tokens(seed, count):
    g = torch.Generator()
    g.manual_seed(seed + 77)
    return torch.randint(0, HYBRID_VOCAB, (count,), generator=g).tolist()


def _prepare_hybrid_prompt(case, seed):
    from qserve_b200.hybrid import StepBatch

    model = _hybrid_model(case, _hybrid_weights(_gen(seed), case))
    lens = _hybrid_lens(case)
    cache = model.new_cache(sum(-(-n // PAGE) * PAGE for n in lens), len(lens), PAGE)
    toks, rows, at = _hybrid_tokens(seed, sum(lens)), [], 0
    for i, n in enumerate(lens):
        cache.admit(i)
        cache.reserve(i, n)
        rows.append((cache.seqs[i].slot, 0, -1, toks[at:at + n]))
        at += n
    return {"model": model, "cache": cache, "batch": StepBatch.build(rows, cache.sync_block_table(), model.device, PAGE)}


def _run_hybrid_prompt(case, s):
    x = s["model"].forward(s["batch"], s["cache"])
    return {"stream": x, **s["cache"].runs[0]}


def _prepare_hybrid_decode(case, seed):
    from qserve_b200.hybrid import StepBatch

    g = _gen(seed)
    model = _hybrid_model(case, _hybrid_weights(g, case))
    B, lens = case["batch"], _lengths(case["batch"], case["ctx"])
    cache = model.new_cache(sum((n + PAGE) // PAGE * PAGE for n in lens), B, PAGE)
    toks, rows = _hybrid_tokens(seed, 2 * B), []
    for i, n in enumerate(lens):
        cache.admit(i)
        cache.reserve(i, n + 1)
        rows.append((cache.seqs[i].slot, n, toks[2 * i], [toks[2 * i + 1]]))
    s = {"model": model, "cache": cache, "batch": StepBatch.build(rows, cache.sync_block_table(), model.device, PAGE)}
    s["scratch"] = torch.empty(max(1, model.scratch_floats(B)), dtype=F32, device="cuda")
    step = lambda: model.logits(model.forward(s["batch"], cache, None, s["scratch"]))
    step()  # eager once, then as the engine replays its decode steps
    torch.cuda.synchronize()
    s["graph"] = torch.cuda.CUDAGraph()
    with torch.cuda.graph(s["graph"]):
        s["logits"] = step()
    _decode_cache(g, case, cache.runs)
    return s


def _run_hybrid_decode(case, s):
    s["graph"].replay()
    runs = s["cache"].runs
    return {"logits": s["logits"], "k": runs[0]["k"], "v": runs[0]["v"], "state": runs[1]["state"], "conv": runs[1]["conv"]}


_KINDS = {"linear": (_prepare_linear, _run_linear), "decode_attention": (_prepare_decode_attention, _run_decode_attention),
          "prompt_attention": (_prepare_prompt_attention, _run_prompt_attention), "prompt_mlp": (_prepare_prompt_mlp, _run_prompt_mlp),
          "decode_layer": (_prepare_decode_layer, _run_decode_layer), "hybrid_attention": (_prepare_hybrid_prompt, _run_hybrid_prompt),
          "hybrid_delta": (_prepare_hybrid_prompt, _run_hybrid_prompt), "hybrid_state_space": (_prepare_hybrid_prompt, _run_hybrid_prompt),
          "hybrid_decode": (_prepare_hybrid_decode, _run_hybrid_decode)}


@torch.no_grad()
def prepare(case, seed):
    return case, _KINDS[case["kind"]][0](case, seed)


@torch.no_grad()
def run(state):
    case, s = state
    return _KINDS[case["kind"]][1](case, s)


# ------------------------------------------------------------------------------------------------------------------------
# work: bytes and operations the path cannot do without
# ------------------------------------------------------------------------------------------------------------------------
def _linear_work(m, n, k, mode):
    weights = n * k + 2 * n if mode == "w8" else n * k // 2 + 4 * n + (2 * n * k // 128 if mode == "grp" else 0)
    return weights + m * k + 2 * m * n + 4 * m, 2 * m * n * k


def _cache_bytes(tokens, hkv, bits):
    return 2 * tokens * hkv * (D * bits // 8 + 4)


def _decode_attention_work(lens, hq, hkv, bits):
    tokens = sum(lens)
    return _cache_bytes(tokens, hkv, bits) + 2 * len(lens) * (2 * hq + 2 * hkv) * D, 4 * tokens * hq * D


def work(case):
    kind = case["kind"]
    if kind == "linear":
        b, f = _linear_work(case["m"], case["n"], case["k"], case["mode"])
        return {"bytes": b, "flops": f}
    if kind.startswith("hybrid"):
        W, H, G = _hybrid_sizes(case["width"])
        lens = _lengths(case["batch"], case["ctx"]) if kind == "hybrid_decode" else _hybrid_lens(case)
        T = len(lens) if kind == "hybrid_decode" else sum(lens)
        att_p, dlt_p = (2 * H + 3 * G + H) * D * W, (2 * G + 3 * H) * D * W + 2 * H * W  # weights: attention, delta
        state, conv = len(lens) * H * D * D, len(lens) * 3 * (2 * G + H) * D
        cell = 3 * G * D * 2  # cache bytes of a position
        if kind == "hybrid_attention":
            pairs = sum(n * (n + 1) // 2 for n in lens)
            return {"bytes": 2 * att_p + 4 * T * W + T * cell, "flops": 2 * T * att_p + pairs * H * 8 * D}
        if kind == "hybrid_delta":
            return {"bytes": 2 * dlt_p + 4 * T * W + 4 * (state + conv), "flops": 2 * T * dlt_p + T * H * D * D * 7}
        if kind == "hybrid_state_space":
            SH, gn = 2 * W // SSM_DIM, 2 * SSM_GROUPS * SSM_STATE
            p = (4 * W + gn + SH) * W + 2 * W * W
            return {"bytes": 2 * p + 4 * T * W + 4 * len(lens) * (SH * SSM_STATE * SSM_DIM + 3 * (2 * W + gn)),
                    "flops": 2 * T * p + T * SH * SSM_STATE * SSM_DIM * 5}
        p = att_p + dlt_p + 6 * HYBRID_FF * W * W + HYBRID_VOCAB * W
        return {"bytes": 2 * p + (sum(lens) + 2 * T) * cell + 8 * (state + conv) + 4 * T * HYBRID_VOCAB,
                "flops": 2 * T * p + (sum(lens) + T) * H * 8 * D + T * H * D * D * 7}
    H, I, hq, hkv = LLAMA[case["model"]][:4]
    if kind == "decode_attention":
        b, f = _decode_attention_work(_lengths(case["batch"], case["ctx"]), hq, hkv, case["bits"])
        return {"bytes": b, "flops": f}
    if kind == "prompt_attention":
        lens = _lengths(case["prompts"], case["ctx"])
        T, pairs = sum(lens), sum(n * (n + 1) // 2 for n in lens)
        b1, f1 = _linear_work(T, (hq + 2 * hkv) * D, H, case["mode"])
        b2, f2 = _linear_work(T, H, hq * D, case["mode"])
        return {"bytes": b1 + b2 + _cache_bytes(T, hkv, case["bits"]) + 2 * T * hq * D, "flops": f1 + f2 + pairs * hq * 4 * D}
    if kind == "prompt_mlp":
        m = case["m"]
        b1, f1 = _linear_work(m, 2 * I, H, case["mode"])
        b2, f2 = _linear_work(m, H, I, case["mode"])
        return {"bytes": b1 + b2 + 2 * m * (2 * H + I), "flops": f1 + f2}
    B = case["batch"]
    total_b, total_f = _decode_attention_work(_lengths(B, case["ctx"]), hq, hkv, case["bits"])
    for n, k in (((hq + 2 * hkv) * D, H), (H, hq * D), (2 * I, H), (H, I)):
        b, f = _linear_work(0, n, k, case["mode"])
        total_b, total_f = total_b + b, total_f + 2 * B * n * k
    return {"bytes": total_b + 2 * B * (3 * H + (hq + 2 * hkv) * D), "flops": total_f}


# ------------------------------------------------------------------------------------------------------------------------
# tolerances: about four times what the paths show against `exact`
# ------------------------------------------------------------------------------------------------------------------------
def tolerance(case):
    kind = case["kind"]
    if kind == "linear":  # integer accumulators, one rounding to fp16
        return {"rel": 1e-3, "max": 4e-3}
    if kind == "decode_attention":  # fp16 operands and outputs; the appended pages are bytes
        return {"rel": 8e-3, "max": 0.1, "differ": 1e-4}
    if kind in ("prompt_attention", "prompt_mlp", "decode_layer"):  # an INT8 code may fall on the other side of a tie between two linear layers
        return {"rel": 3e-2, "max": 0.3, "differ": 1e-3}
    return {"rel": 1.6e-2, "max": 0.5}  # bf16 operands


# ------------------------------------------------------------------------------------------------------------------------
# the same numbers in plain torch, 64 bits
# ------------------------------------------------------------------------------------------------------------------------
def _unpack(w):
    """Weights [n, k] in 64 bits.  INT4 layout: 32 x 32 tiles of 32 lanes x 16 bytes; lane c * 4 + e, byte d * 8 + b * 4 + f holds row b * 8 + c (low
    nibble) and row b * 8 + c + 16 (high nibble), column d * 16 + e * 4 + f.  Level-2 numbers: place c * 4 + j of 32 belongs to row j * 8 + c."""
    if w["mode"] == "w8":
        return w["w"].to(F64)
    n, k = w["w"].shape[0], w["w"].shape[1] * 2
    p = w["w"].view(torch.uint8).view(n // 32, k // 32, 8, 4, 2, 2, 4)  # [.., .., c, e, d, b, f]
    q = torch.stack([p & 15, p >> 4], 0)                               # [half, n32, k32, c, e, d, b, f]
    q = q.permute(1, 0, 6, 3, 2, 5, 4, 7).reshape(n, k).to(F64)
    if w["mode"] == "chn":
        return q
    flat = lambda t: t.view(-1, n // 32, 8, 4).permute(0, 1, 3, 2).reshape(-1, n).t().to(F64)
    return (q.view(n, k // 128, 128) * flat(w["s2"])[:, :, None] + flat(w["z2"])[:, :, None]).view(n, k)


def _linear64(w, q, scale, asum):
    acc = q.to(F64) @ _unpack(w).t()
    out = acc * w["s"].to(F64) * scale.to(F64)[:, None]
    return out - w["sz"].to(F64) * asum.to(F64)[:, None] if w["mode"] == "chn" else out


def _quant64(x):
    """Codes, and scale and row sum as the operators hand them on: fp16 numbers."""
    amax = x.abs().amax(-1)
    return torch.round(x * (127.0 / amax)[:, None]), (amax / 127.0).to(HALF), x.sum(-1).to(HALF)


def _norm64(x, gamma, eps):
    d = x - x.mean(-1, keepdim=True)
    return d * torch.rsqrt((d * d).mean(-1, keepdim=True) + eps) * gamma.to(F64)


def _rope64(x, pos, base):
    """x [T, heads, D] at positions pos [T]: pairs (i, i + D / 2)."""
    f = base ** (-torch.arange(0, D, 2, dtype=F64, device=x.device) / D)
    a = pos.to(F64)[:, None, None] * f
    c, s, lo, hi = torch.cos(a), torch.sin(a), x[..., :D // 2], x[..., D // 2:]
    return torch.cat([lo * c - hi * s, hi * c + lo * s], -1)


def _cached64(pool, rows, n, hkv, bits):
    """Positions 0 .. n - 1 of a sequence out of its pages: [n, hkv, D]."""
    code = hkv * PAGE * D * bits // 8
    p = pool[rows]
    c = p[:, :code].reshape(-1, hkv, PAGE, D * bits // 8)
    if bits == 4:
        c = torch.stack([c & 15, c >> 4], -1).flatten(-2)
    meta = p[:, code:].reshape(-1).view(HALF).view(-1, 2, hkv, PAGE, 1).to(F64)
    return (meta[:, 0] * (c.to(F64) - meta[:, 1])).permute(0, 2, 1, 3).reshape(-1, hkv, D)[:n]


def _decode_attention64(s, qkv, bits):
    hq, hkv = s["hq"], s["hkv"]
    pos = s["lens"].long() - 1
    q, k, v = (t.reshape(len(pos), -1, D) for t in qkv.split([hq * D, hkv * D, hkv * D], -1))
    q, k = _rope64(q, pos, s["base"]), _rope64(k, pos, s["base"])
    outs = []
    for i, n in enumerate(pos.tolist()):
        K = torch.cat([_cached64(s["pools"][0], s["pages"][i], n, hkv, bits), k[i][None]])
        V = torch.cat([_cached64(s["pools"][1], s["pages"][i], n, hkv, bits), v[i][None]])
        a = torch.softmax(torch.einsum("gjd,ngd->gjn", q[i].view(hkv, hq // hkv, D), K) * D ** -0.5, -1)
        outs.append(torch.einsum("gjn,ngd->gjd", a, V).reshape(hq, D))
    return torch.stack(outs)


def _exact_quantised(case, seed):
    s = _KINDS[case["kind"]][0](dict(case), seed)
    kind = case["kind"]
    if kind == "linear":
        return _linear64(s["lin"], s["x"], s["scale"], s["sum"])
    if kind == "decode_attention":
        return {"out": _decode_attention64(s, s["qkv"].to(F64), case["bits"]), "k": None, "v": None}
    if kind == "prompt_attention":
        hq, hkv = s["hq"], s["hkv"]
        qkv = _linear64(s["lin"]["qkv"], s["x"], s["scale"], s["sum"])
        lens = s["lens"].tolist()
        pos = torch.cat([torch.arange(n, device="cuda") for n in lens])
        q, k, v = (t.reshape(s["T"], -1, D) for t in qkv.split([hq * D, hkv * D, hkv * D], -1))
        q, k = _rope64(q, pos, s["base"]), _rope64(k, pos, s["base"])
        a, at = torch.empty(s["T"], hq, D, dtype=F64, device="cuda"), 0
        for n in lens:
            mask = torch.full((n, n), -math.inf, dtype=F64, device="cuda").triu(1)
            for h in range(hq):
                g = h // (hq // hkv)
                w = torch.softmax(q[at:at + n, h] @ k[at:at + n, g].t() * D ** -0.5 + mask, -1)
                a[at:at + n, h] = w @ v[at:at + n, g]
            at += n
        out = _linear64(s["lin"]["o"], *_quant64(a.flatten(1)))
        return {"out": out, "attention": a, "qkv": torch.cat([q.flatten(1), k.flatten(1), v.flatten(1)], 1), "k": None, "v": None}
    if kind == "prompt_mlp":
        x = s["x"].to(F64)
        gu = _linear64(s["gate_up"], *_quant64(_norm64(x, s["gamma"], s["eps"])))
        gate, up = gu.chunk(2, -1)
        act = gate * torch.sigmoid(gate) * up
        return {"out": x + _linear64(s["down"], *_quant64(act)), "act": act, "codes": None}
    x, w = s["x"].to(F64), s["w"]
    qkv = _linear64(w["qkv"], *_quant64(_norm64(x, s["gamma"][0], s["eps"])))
    a = _decode_attention64(s, qkv, case["bits"])
    h = x + _linear64(w["o"], *_quant64(a.flatten(1)))
    gate, up = _linear64(w["gate_up"], *_quant64(_norm64(h, s["gamma"][1], s["eps"]))).chunk(2, -1)
    y = h + _linear64(w["down"], *_quant64(gate * torch.sigmoid(gate) * up))
    return {"hidden": y, "middle": h, "qkv": qkv, "k": None, "v": None}


def _unit64(x):
    return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + EPS)


def _pairs64(x, pos):
    """Interleaved rotary pairs on the first half of a head, YaRN-blended frequencies (factor 4 over 4096 positions, ramp 32 .. 1 turns)."""
    dims, base, factor, orig, fast, slow = D // 2, 1e6, 4.0, 4096.0, 32.0, 1.0
    i = torch.arange(dims // 2, dtype=F64, device=x.device)
    turn = lambda t: dims * math.log(orig / (2 * math.pi * t)) / (2 * math.log(base))
    lo, hi = max(math.floor(turn(fast)), 0), min(math.ceil(turn(slow)), dims - 1)
    ramp = ((i - lo) / max(hi - lo, 0.001)).clamp(0, 1)
    f = base ** (-2 * i / dims)
    a = pos.to(F64)[:, None, None] * (f / factor * ramp + f * (1 - ramp))
    amp = 0.1 * math.log(factor) + 1.0
    c, s, u, v = torch.cos(a) * amp, torch.sin(a) * amp, x[..., 0:dims:2], x[..., 1:dims:2]
    out = x.clone()
    out[..., 0:dims:2], out[..., 1:dims:2] = u * c - v * s, v * c + u * s
    return out


def _diff_lambda(w, p):
    dot = lambda a, b: float((w[p + a] * w[p + b]).sum())
    return math.exp(dot("lq1", "lk1")) - math.exp(dot("lq2", "lk2")) + 0.5


def _attention64(h, pos, spans, w, p, H, G, cached=None):
    """Differential attention of rows h; spans: rows of each sequence; cached: earlier (keys, values) of each sequence.  Returns the mixer's output
    and the new keys and values."""
    q = _pairs64((h @ w[p + "q"].t()).view(-1, H * 2, D), pos).view(-1, H, 2, D)
    k = _pairs64((h @ w[p + "k"].t()).view(-1, G * 2, D), pos).view(-1, G, 2, D)
    v = (h @ w[p + "v"].t()).view(-1, G, D)
    lam, out = _diff_lambda(w, p), torch.empty(h.shape[0], H, D, dtype=F64, device=h.device)
    for i, (a, b) in enumerate(spans):
        K, V = (k[a:b], v[a:b]) if cached is None else (torch.cat([cached[i][0], k[a:b]]), torch.cat([cached[i][1], v[a:b]]))
        n, m = K.shape[0], b - a
        mask = torch.full((m, n), -math.inf, dtype=F64, device=h.device).triu(n - m + 1)
        for hd in range(H):
            g = hd // (H // G)
            r = [torch.softmax(q[a:b, hd, j] @ K[:, g, j].t() * D ** -0.5 + mask, -1) @ V[:, g] for j in range(2)]
            out[a:b, hd] = _unit64(r[0] - lam * r[1]) * 0.5
    return out.flatten(1), k, v


def _conv64(x, before, taps):
    n, t = x.shape[0], taps.shape[1]
    pad = torch.cat([before, x])
    return sum(pad[j:j + n] * taps[:, j] for j in range(t)), pad[n:]


def _scan64(steps, S, lens, step):
    """step(S, t, rows) for t = 0 .. max(lens) - 1, where the sequences that have ended keep their state."""
    for t in range(steps):
        S = step(S, t, torch.tensor([t < n for n in lens], device=S.device))
    return S


def _padded(x, spans, steps):
    out = torch.zeros(len(spans), steps, *x.shape[1:], dtype=F64, device=x.device)
    for i, (a, b) in enumerate(spans):
        out[i, :b - a] = x[a:b]
    return out


def _unpadded(x, spans):
    return torch.cat([x[i, :b - a] for i, (a, b) in enumerate(spans)])


def _delta64(h, spans, w, p, H, G, S, before):
    lens = [b - a for a, b in spans]
    x = torch.cat([h @ w[p + n].t() for n in ("q", "k", "v")], 1)
    taps = torch.cat([w[p + n + ".conv"] for n in ("q", "k", "v")], 0)
    c = [_conv64(x[a:b], before[i], taps) for i, (a, b) in enumerate(spans)]
    y = torch.cat([t[0] for t in c])
    y = y * torch.sigmoid(y)
    q, k, v = (t.reshape(h.shape[0], -1, D) for t in y.split([G * D, G * D, H * D], 1))
    unit = lambda t: t * torch.rsqrt((t * t).sum(-1, keepdim=True) + 1e-6)
    beta = torch.sigmoid(h @ w[p + "b"].t())
    decay = torch.exp(-torch.exp(w[p + "A_log"]) * torch.nn.functional.softplus(h @ w[p + "a"].t() + w[p + "dt_bias"]))
    steps = max(lens)
    q, k, v, beta, decay = (_padded(t, spans, steps) for t in ((unit(q) * D ** -0.5).repeat_interleave(H // G, 1), unit(k).repeat_interleave(H // G, 1),
                                                               v, beta, decay))
    out = torch.zeros(len(spans), steps, H, D, dtype=F64, device=h.device)

    def step(S, t, live):
        N = S * decay[:, t, :, None, None]
        u = beta[:, t, :, None] * (v[:, t] - torch.einsum("bhdv,bhd->bhv", N, k[:, t]))
        N = N + k[:, t, :, :, None] * u[:, :, None, :]
        out[:, t] = torch.einsum("bhdv,bhd->bhv", N, q[:, t])
        return torch.where(live[:, None, None, None], N, S)

    S = _scan64(steps, S, lens, step)
    gate = h @ w[p + "g"].t()
    o = _unit64(_unpadded(out, spans)) * w[p + "norm"] * (gate * torch.sigmoid(gate)).view(-1, H, D)
    return o.flatten(1), S, torch.stack([t[1] for t in c])


def _state_space64(h, spans, w, p, W):
    H, N, P, G = 2 * W // SSM_DIM, SSM_STATE, SSM_DIM, SSM_GROUPS
    lens, inner = [b - a for a, b in spans], 2 * W
    z, xbc, dt = (h @ w[p + "in"].t()).split([inner, inner + 2 * G * N, H], 1)
    zero = torch.zeros(SSM_CONV - 1, xbc.shape[1], dtype=F64, device=h.device)
    c = [_conv64(xbc[a:b], zero, w[p + "conv"]) for a, b in spans]
    y = torch.cat([t[0] for t in c]) + w[p + "conv.b"]
    x, B, C = (y * torch.sigmoid(y)).split([inner, G * N, G * N], 1)
    dt = torch.nn.functional.softplus(dt + w[p + "dt_bias"])
    x, B, C = x.reshape(-1, H, P), B.reshape(-1, G, N).repeat_interleave(H // G, 1), C.reshape(-1, G, N).repeat_interleave(H // G, 1)
    steps = max(lens)
    xs, Bs, Cs, dts = (_padded(t, spans, steps) for t in (x, B, C, dt))
    a = torch.exp(-torch.exp(w[p + "A_log"]) * dts)
    out = torch.zeros(len(spans), steps, H, P, dtype=F64, device=h.device)

    def step(S, t, live):
        M = S * a[:, t, :, None, None] + Bs[:, t, :, :, None] * (dts[:, t, :, None] * xs[:, t])[:, :, None, :]
        out[:, t] = torch.einsum("bhnp,bhn->bhp", M, Cs[:, t])
        return torch.where(live[:, None, None, None], M, S)

    S = _scan64(steps, torch.zeros(len(spans), H, N, P, dtype=F64, device=h.device), lens, step)
    y = ((_unpadded(out, spans) + w[p + "D"][:, None] * x).flatten(1)) * z * torch.sigmoid(z)
    y = _unit64(y.view(-1, SSM_GROUPS, inner // SSM_GROUPS)).flatten(1) * w[p + "norm"]
    return y, S, torch.stack([t[1] for t in c])


def _embed64(w, toks, prevs, scale=1.0):
    x = w["embed"][toks] * scale
    if "bigram" not in w:
        return x
    row = torch.where(prevs < 0, torch.full_like(toks, BUCKETS), (prevs * MUL_PREV + toks * MUL_CUR) % BUCKETS)
    return x + w["bigram"][row]


def _exact_hybrid_prompt(case, seed):
    W, H, G = _hybrid_sizes(case["width"])
    w = {k: v.to(F64) for k, v in _hybrid_weights(_gen(seed), case).items()}
    lens = _hybrid_lens(case)
    toks = torch.tensor(_hybrid_tokens(seed, sum(lens)), device="cuda")
    spans, at = [], 0
    for n in lens:
        spans.append((at, at + n))
        at += n
    prevs = toks.roll(1)
    prevs[[a for a, _ in spans]] = -1
    pos = torch.cat([torch.arange(n, device="cuda") for n in lens])
    p = "l0.mix."
    if case["kind"] == "hybrid_state_space":
        x = _embed64(w, toks, prevs, 8.0)
        y, S, c = _state_space64(_unit64(x) * w["l0.norm1"], spans, w, p, W)
        return {"stream": x + y @ w[p + "o"].t(), "state": S, "conv": c}
    x = _embed64(w, toks, prevs)
    h = _unit64(x) * (1.0 + w["l0.norm1"])
    if case["kind"] == "hybrid_attention":
        y, k, v = _attention64(h, pos, spans, w, p, H, G)
        return {"stream": x + y @ w[p + "o"].t(), "k": None, "v": None}
    S = torch.zeros(len(lens), H, D, D, dtype=F64, device="cuda")
    before = torch.zeros(len(lens), 3, (2 * G + H) * D, dtype=F64, device="cuda")
    y, S, c = _delta64(h, spans, w, p, H, G, S, before)
    return {"stream": x + y @ w[p + "o"].t(), "state": S, "conv": c}


def _exact_hybrid_decode(case, seed):
    s = _prepare_hybrid_decode(case, seed)
    W, H, G = _hybrid_sizes(case["width"])
    w = {k: v.to(F64) for k, v in _hybrid_weights(_gen(seed), case).items()}
    B, lens = case["batch"], _lengths(case["batch"], case["ctx"])
    both = torch.tensor(_hybrid_tokens(seed, 2 * B), device="cuda").view(B, 2)
    runs, table = s["cache"].runs, s["cache"].block_table
    slots = torch.tensor([s["cache"].seqs[i].slot for i in range(B)], device="cuda")
    spans = [(i, i + 1) for i in range(B)]
    cached = []
    for i, n in enumerate(lens):
        pages = table[slots[i], :-(-(n + 1) // PAGE)].long()
        cached.append((runs[0]["k"][pages].reshape(-1, G, 2, D)[:n].to(F64), runs[0]["v"][pages].reshape(-1, G, D)[:n].to(F64)))
    x = _embed64(w, both[:, 1], both[:, 0])
    norm = lambda t, n: _unit64(t) * (1.0 + w[n])
    ff = lambda t, q: (torch.nn.functional.gelu(t @ w[q + "gate"].t(), approximate="tanh") * (t @ w[q + "up"].t())) @ w[q + "down"].t()
    y, _, _ = _attention64(norm(x, "l0.norm1"), torch.tensor(lens, device="cuda"), spans, w, "l0.mix.", H, G, cached)
    x = x + y @ w["l0.mix.o"].t() + ff(norm(x, "l0.norm2"), "l0.mlp.")
    y, S, c = _delta64(norm(x, "l1.norm1"), spans, w, "l1.mix.", H, G, runs[1]["state"][slots].to(F64), runs[1]["conv"][slots].to(F64))
    x = x + y @ w["l1.mix.o"].t() + ff(norm(x, "l1.norm2"), "l1.mlp.")
    state, conv = runs[1]["state"].to(F64), runs[1]["conv"].to(F64)
    state[slots], conv[slots] = S, c
    return {"logits": norm(x, "final.norm") @ w["head"].t(), "k": None, "v": None, "state": state, "conv": conv}


@torch.no_grad()
def exact(case, seed):
    if case["kind"] == "hybrid_decode":
        return _exact_hybrid_decode(case, seed)
    if case["kind"].startswith("hybrid"):
        return _exact_hybrid_prompt(case, seed)
    return _exact_quantised(case, seed)
