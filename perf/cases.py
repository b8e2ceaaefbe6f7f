"""The work a user of this library has it do: one pass of a mixture-of-experts layer, decode windows and prompts.

A decode case is one step of a resident layer over a window of 1 to 64 tokens (moe.NativeMoELayer: the whole step behind one
call, issued directly or replayed as a CUDA graph; moe.MoELayer: the same step call by call, as an engine that drops the
operators in issues it).  A prompt case is one pass of moe.PrefillMoELayer over 65 to 16,384 rows.  A case names the layer's
widths, its router, the experts' block format, the rows and their type; weights and rows are made from the seed alone.
"""
import math

import torch

from basalt_b200 import capi, moe, pack

# The layers of this repository's benchmark, tests and defaults: n_embd, n_ff, experts, top-k, router kind, groups, kept groups, scale.
SHAPES = {
    "flash": (2048, 512, 512, 10, "softmax", 1, 1, 1.0),        # the benchmark's flash-next-style layer
    "flash-wide": (2560, 640, 512, 10, "softmax", 1, 1, 1.0),   # the same at the widths that no 256-column plane fits (640)
    "v41": (5120, 2304, 384, 6, "sqrt_softplus", 1, 1, 1.5),    # the router's defaults
    "deepseek": (7168, 2048, 256, 8, "sigmoid", 8, 4, 2.5),     # the benchmark's DeepSeek-style layer
    "small": (2048, 512, 64, 8, "softmax", 1, 1, 1.0),          # the CPU reference configuration
}
GATES = {"softmax": capi.GATE_SOFTMAX, "sigmoid": capi.GATE_SIGMOID, "sqrt_softplus": capi.GATE_SQRT_SOFTPLUS}
Q6_K, IQ3_S, IQ1_M, NVFP4 = capi.TYPE_Q6_K, 21, capi.TYPE_IQ1_M, capi.TYPE_NVFP4
# experts' format -> (routed type, shared expert's type or None, blobs repacked into planes at load)
FORMATS = {"nvfp4": (NVFP4, NVFP4, True), "nvfp4-in-place": (NVFP4, NVFP4, False), "q6_k": (Q6_K, Q6_K, False),
           "iq1_m": (IQ1_M, Q6_K, False), "iq3_s": (IQ3_S, Q6_K, False)}
SIGMA = 0.02            # standard deviation of the weights
POOL_ROWS = 2048        # distinct quantised rows a layer's matrices are dealt from


def _case(name, kind, shape, fmt, tokens, act="bf16", api="native", graph=False, norm=False, residual=False, shared=True):
    return dict(name=name, kind=kind, shape=shape, format=fmt, tokens=tokens, act=act, api=api, graph=graph, norm=norm, residual=residual, shared=shared)


def listed():
    return [
        # one user's next token: launches and latency, an engine that replays its step as a graph
        _case("decode-1-nvfp4", "decode", "flash", "nvfp4", 1, graph=True),
        # a few streams, issued without a graph, the layer taking the un-normed fp32 residual stream and adding it back
        _case("decode-8-nvfp4-norm", "decode", "flash", "nvfp4", 8, act="f32", norm=True, residual=True),
        # a full serving window on the layer the benchmark quotes
        _case("decode-64-nvfp4", "decode", "flash", "nvfp4", 64, graph=True),
        # the same window where one expert is 25 MB: the weight stream at its longest
        _case("decode-64-nvfp4-deepseek", "decode", "deepseek", "nvfp4", 64, graph=True),
        # an odd window over blobs used as the file holds them, operator by operator
        _case("decode-27-nvfp4-in-place", "decode", "flash-wide", "nvfp4-in-place", 27, api="calls"),
        # the low-bit codebook layer with its 6-bit shared expert
        _case("decode-64-iq1m", "decode", "deepseek", "iq1_m", 64),
        # the K-quant layer of the CPU reference configuration
        _case("decode-16-q6k", "decode", "small", "q6_k", 16),
        # a speculative window on the 3-bit codebook format
        _case("decode-5-iq3s", "decode", "flash", "iq3_s", 5),
        # a long prompt over many small experts
        _case("prompt-16384-nvfp4", "prompt", "flash", "nvfp4", 16384),
        # a short, ragged prompt of fp32 rows: a couple of tiles an expert, most of them not full
        _case("prompt-777-nvfp4-v41", "prompt", "v41", "nvfp4", 777, act="f32"),
        # a long prompt over large experts
        _case("prompt-8192-nvfp4-deepseek", "prompt", "deepseek", "nvfp4", 8192),
        # a prompt over codebook blobs read in place
        _case("prompt-4096-iq1m", "prompt", "deepseek", "iq1_m", 4096, shared=False),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    act = rng.choice(("bf16", "f32"))
    if rng.random() < 0.6:
        fmt = rng.choices(("nvfp4", "nvfp4-in-place", "q6_k", "iq1_m", "iq3_s"), (50, 10, 10, 15, 15))[0]
        shape = rng.choice({"nvfp4": ("flash", "v41", "deepseek"), "nvfp4-in-place": ("flash", "flash-wide"), "q6_k": ("small", "flash"),
                            "iq1_m": ("v41", "deepseek"), "iq3_s": ("small", "flash")}[fmt])
        c = _case("", "decode", shape, fmt, _log_int(rng, 1, 64), act=act)
        how = rng.choice(("graph", "direct", "norm", "calls"))
        c["graph"] = how == "graph"
        c["norm"] = c["residual"] = how == "norm"
        if how == "calls":
            c["api"] = "calls"
    else:
        fmt = rng.choices(("nvfp4", "nvfp4-in-place", "q6_k", "iq1_m"), (60, 10, 10, 20))[0]
        shape, most = rng.choice({"nvfp4": (("flash", 16384), ("v41", 8192), ("deepseek", 8192)), "nvfp4-in-place": (("flash", 16384), ("flash-wide", 8192)),
                                  "q6_k": (("small", 4096), ("flash", 4096)), "iq1_m": (("v41", 4096), ("deepseek", 4096))}[fmt])
        c = _case("", "prompt", shape, fmt, _log_int(rng, 65, most), act=act, shared=fmt != "iq1_m")
    del c["name"]
    return c


# ---------------------------------------------------------------------------------------------------------------- inputs
def _f16_bytes(v):
    """fp16 values [...] -> their bytes [..., 2]"""
    return v.half().contiguous().view(torch.uint8).reshape(*v.shape, 2)


def _q6k_rows(w):
    """fp32 [rows][cols] -> Q6_K blocks: a scale per 16 values from its largest magnitude, int8 scales under one fp16 d per 256"""
    rows, cols = w.shape
    g = w.reshape(rows, cols // 256, 16, 16)
    s = g.abs().amax(-1) / 31.0
    d = (s.amax(-1) / 127.0).clamp_min(1e-7).half()
    sc = (s / d.float()[..., None]).round().clamp_(1, 127)
    q = ((g / (d.float()[..., None] * sc)[..., None]).round().clamp_(-32, 31) + 32).to(torch.uint8).reshape(rows, cols // 256, 2, 4, 32)
    ql = (q[:, :, :, :2] & 15) | ((q[:, :, :, 2:] & 15) << 4)
    qh = (q[:, :, :, 0] >> 4) | ((q[:, :, :, 1] >> 4) << 2) | ((q[:, :, :, 2] >> 4) << 4) | ((q[:, :, :, 3] >> 4) << 6)
    n = (rows, cols // 256)
    return torch.cat([ql.reshape(*n, 128), qh.reshape(*n, 64), sc.to(torch.int8).view(torch.uint8).reshape(*n, 16), _f16_bytes(d)], -1).reshape(rows, -1)


def _codebook_rows(rows, cols, block, g):
    """random valid blocks of a codebook format: uniform codes under a scale that gives weights of about SIGMA"""
    raw = torch.randint(0, 256, (rows, cols // 256, block), generator=g, device="cuda", dtype=torch.uint8)
    u = 1.0 + torch.rand((rows, cols // 256), generator=g, device="cuda")
    if block == 56:        # IQ1_M: d (2 s + 1) (g +- 1/8); the bits of d in the top nibbles of the four scale words
        bits = _f16_bytes(u * 0.0022)
        for j in range(4):
            nib = (bits[..., j >> 1] >> (4 * (j & 1))) & 15
            raw[..., 49 + 2 * j] = (raw[..., 49 + 2 * j] & 15) | (nib << 4)
    else:                  # IQ3_S: d (2 s + 1) x odd magnitude up to 15
        raw[..., :2] = _f16_bytes(u * 0.000105)
    return raw.reshape(rows, -1)


def _rows(t, rows, cols, g):
    if t in (IQ1_M, IQ3_S):
        return _codebook_rows(rows, cols, 56 if t == IQ1_M else 110, g)
    w = torch.randn((rows, cols), generator=g, device="cuda") * SIGMA
    if t == Q6_K:
        return _q6k_rows(w)
    return pack.quantize_nvfp4(w / (5.0 * SIGMA / (6.0 * 448.0)))     # under the fp32 scale of a matrix whose largest weight is 5 sigma


def _blobs(t, n, H, I, g):
    """n expert blobs: every row of every matrix dealt from a pool of quantised rows"""
    L = moe.native_expert_layout(t, t, H, I)
    out = torch.zeros((n, (L.bytes + 15) // 16 * 16), dtype=torch.uint8, device="cuda")
    for at, per, width in ((0, 2 * I, H), (L.down_off, H, I)):
        pool = _rows(t, POOL_ROWS, width, g)
        unit = torch.int32 if pool.shape[1] % 4 == 0 and out.shape[1] % 4 == 0 and at % 4 == 0 else torch.int16
        pool, dst = pool.view(unit), out.view(unit)
        size = torch.empty((), dtype=unit).element_size()
        a, b = at // size, (at + per * pool.shape[1] * size) // size
        for e in range(0, n, 64):
            m = min(64, n - e)
            dst[e:e + m, a:b] = pool[torch.randint(0, POOL_ROWS, (m * per,), generator=g, device="cuda")].view(m, -1)
    if t == NVFP4:
        tail = torch.tensor([5.0 * SIGMA / (6.0 * 448.0)] * 3 + [0.0], device="cuda")
        out[:, L.bytes - 16:L.bytes] = tail.view(torch.uint8)
    return L, out


def prepare(case, seed):
    H, I, E, k, gate_kind, n_group, kept, scale = SHAPES[case["shape"]]
    t, shared_t, packed = FORMATS[case["format"]]
    g = torch.Generator(device="cuda").manual_seed(seed)
    T, prompt = case["tokens"], case["kind"] == "prompt"
    gate = torch.randn((E, H), generator=g, device="cuda") * SIGMA
    bias = torch.randn(E, generator=g, device="cuda") * 0.01 if gate_kind != "softmax" else None
    args = moe.RouterArgs(n_expert=E, n_embd=H, k=k, weight_scale=scale, gate=GATES[gate_kind], n_group=n_group, topk_group=kept)
    own_shared = case["shared"] and shared_t != t and not prompt
    L, blobs = _blobs(t, E + (1 if case["shared"] and not own_shared else 0), H, I, g)
    if packed:
        blobs = moe.pack_experts(L, blobs)
    shared_L = shared = None
    if own_shared:
        shared_L, s = _blobs(shared_t, 1, H, I, g)
        shared = s[0]
    elif case["shared"]:
        shared = blobs[E]
    # hidden states share a component, which makes some experts more popular than others
    x = torch.randn((T, H), generator=g, device="cuda") + 0.5 * torch.randn(H, generator=g, device="cuda")
    x = x.bfloat16() if case["act"] == "bf16" else x
    norm_w = 1.0 + 0.1 * torch.randn(H, generator=g, device="cuda") if case["norm"] else None
    if prompt:
        layer = moe.PrefillMoELayer(gate, bias, blobs[:E], L, args, shared_blob=shared, max_tokens=T, packed=packed)
    elif case["api"] == "calls":
        layer = moe.MoELayer(gate, bias, blobs[:E], L, args, shared_blob=shared, shared_layout=shared_L, max_tokens=T, packed=packed, norm_w=norm_w)
    else:
        layer = moe.NativeMoELayer(gate, bias, blobs[:E], L, args, shared_blob=shared, shared_layout=shared_L, max_tokens=T, packed=packed, norm_w=norm_w)
    if case["graph"]:
        layer.capture(x)
    residual = torch.randn((T, H), generator=g, device="cuda") if case["residual"] else None
    return dict(case=case, layer=layer, x=x, residual=residual, keep=(gate, bias, blobs, shared, norm_w))


def run(state):
    case, layer = state["case"], state["layer"]
    if case["graph"]:
        y = layer.forward_graphed(state["x"])
    elif state["residual"] is not None:
        y = layer.forward(state["x"], state["residual"])
    else:
        y = layer.forward(state["x"])
    out = dict(y=y, logits=layer.logits, ids=layer.ids, weights=layer.w)
    if getattr(layer, "status", None) is not None:
        out["status"] = layer.status       # 0: no wait inside a kernel gave up
    return out


# ---------------------------------------------------------------------------------------------------------------- measure
def work(case):
    """Every touched expert's blob once, the gate matrix, the rows in and the results out; two operations a weight and row."""
    H, I, E, k = SHAPES[case["shape"]][:4]
    t, shared_t, _ = FORMATS[case["format"]]
    T, sh = case["tokens"], 1 if case["shared"] else 0
    touched = E * (1.0 - (1.0 - k / E) ** T)
    size = touched * moe.native_expert_layout(t, t, H, I).bytes
    if sh:
        s = t if case["kind"] == "prompt" else shared_t
        size += moe.native_expert_layout(s, s, H, I).bytes
    size += E * H * 4 + T * (H * (2 if case["act"] == "bf16" else 4) + H * 4 * (2 if case["residual"] else 1) + E * 4 + k * 8)
    return {"bytes": size, "flops": 2.0 * T * (3.0 * H * I * (k + sh) + E * H)}


def tolerance(case):
    """About four times what was measured against the same layer in 64 bits (NVFP4 planes: four FP4 terms a row, 1.4e-4 .. 1.8e-4;
    prompts over blobs in place: fp16 rows, 2.1e-4 where the rows are bf16 and 3.6e-4 where they are rounded too; NVFP4 decode in
    place: fp32-class, 0.2e-6 .. 1.6e-6) and against fp32 products (two int8 terms a row, 1e-4).  A prompt's logits come from a
    tensor-core product, so two experts may tie in them."""
    packed = FORMATS[case["format"]][2]
    if case["kind"] == "prompt":
        return {"rel": 7e-4 if packed else 8e-4 if case["act"] == "bf16" else 1.4e-3, "differ": 1e-4}
    return {"rel": {"nvfp4": 7e-4, "nvfp4-in-place": 1e-5}.get(case["format"], 4e-4)}
