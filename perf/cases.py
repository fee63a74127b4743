"""The work whose time counts: decode steps of Qwen3 dense models and the operators they are made of, each called
through the operator API the way a serving loop or an operator-level user calls it (eager calls on the current
stream, weights and caches resident on the GPU).

A case is a dict of plain values.  ``op`` picks the entry point, the rest are its sizes:

``gemv``       ``GemvOp``                y[N] = W[N, K] . x[K]
``rmsnorm``    ``RmsNormOp``             rows of activations, bf16 with weight or fp32 without
``qk_rope``    ``FusedQkNormRopeOp``     head norm, rotation and cache write of one decode step, one position per row
``attn``       ``AttnDecodeOp``          split-KV grouped-query attention, rows of one length or ragged
``ffn``        ``FusedOProjFfnOp``       output projection, SwiGLU FFN and both residuals
``layer``      ``Qwen3DenseDecodeOp``    one whole decode layer, the new k / v written into the cache
``stack``      ``Qwen3DecodeStackOp``    several layers in one call with norm weights and RoPE; rows of one length,
                                         ragged (``ragged``) or ragged over page pools (``page``)

Sizes: the model shapes of ``ezops_b200.workloads``, batch 1 to 64, context 64 to 8192.  Inputs follow that module's
distributions (activations and KV N(0, 1), projections N(0, 0.02), norm weights 1 + N(0, 0.1)), drawn on the GPU from
the seed.
"""

from __future__ import annotations

import torch

import ezops_b200 as ez
from ezops_b200 import workloads as wl

BF16 = torch.bfloat16
SHAPES = {s.name: s for s in (wl.QWEN3_0_6B, wl.QWEN3_VL_2B, wl.QWEN3_8B, wl.QWEN3_32B)}
LARGEST_BYTES = 3.2e9  # what the largest listed case moves; drawn cases stay below


def listed():
    return [
        # One projection of one token: the smallest unit of work, launch latency and one pass over 34 MB of weights.
        dict(name="gemv_4096", op="gemv", N=4096, K=4096),
        # The hidden-state norm of a batch of 32 tokens: a call of a few microseconds.
        dict(name="rmsnorm_32x4096", op="rmsnorm", rows=32, dim=4096, dtype="bf16"),
        # q / k norm, RoPE and cache write for 32 tokens at 32 different positions.
        dict(name="qk_rope_32tok", op="qk_rope", B=32, NQ=32, NKV=8, D=128, S=8192),
        # Attention of 32 sequences whose lengths are spread over 1024 .. 8192: a full continuous batch.
        dict(name="attn_b32_ragged", op="attn", B=32, H=32, NKV=8, D=128, S=8192, min_len=1024),
        # The tail of a layer for one token, for programs that run their own attention.
        dict(name="ffn_8b_b1", op="ffn", model="qwen3-8b", B=1),
        # The smallest model and a short prompt of odd length: nothing but latency.
        dict(name="layer_06b_b1", op="layer", model="qwen3-0.6b", B=1, S=301),
        # One token of one user, the headline configuration.
        dict(name="layer_8b_b1", op="layer", model="qwen3-8b", B=1, S=4096),
        # A handful of users.
        dict(name="layer_8b_b8", op="layer", model="qwen3-8b", B=8, S=4096),
        # A busy server: the batch where projections become skinny GEMMs.
        dict(name="layer_8b_b32", op="layer", model="qwen3-8b", B=32, S=4096),
        # The largest: full batch, long context, the large model.
        dict(name="layer_32b_b64", op="layer", model="qwen3-32b", B=64, S=8192),
        # A whole decode step of the small model (28 layers) for four users whose contexts differ.
        dict(name="stack_06b_b4_ragged", op="stack", model="qwen3-0.6b", B=4, S=1024, layers=28, ragged=True, page=0),
        # Eight layers (one pipeline stage) of the 2B model for an odd batch over paged caches.
        dict(name="stack_vl2b_b13_paged", op="stack", model="qwen3-vl-2b", B=13, S=1024, layers=8, ragged=True, page=256),
    ]


def _log_int(rng, lo, hi):
    """An integer spread evenly over the logarithm of [lo, hi]."""
    return min(hi, max(lo, int(round(lo * (hi / lo) ** rng.random()))))


def draw(rng):
    while True:
        case = _draw_any(rng)
        if work(case)["bytes"] <= LARGEST_BYTES:
            return case


def _draw_any(rng):
    op = rng.choice(["gemv", "rmsnorm", "qk_rope", "attn", "ffn", "layer", "layer", "layer", "stack", "stack"])
    model = rng.choice(list(SHAPES))
    B = _log_int(rng, 1, 64)
    if op == "gemv":
        return dict(op=op, N=_log_int(rng, 64, 32768), K=16 * _log_int(rng, 16, 1600))
    if op == "rmsnorm":
        return dict(op=op, rows=_log_int(rng, 1, 512), dim=8 * _log_int(rng, 16, 2048), dtype=rng.choice(["bf16", "fp32"]))
    if op == "qk_rope":
        sh = SHAPES[model]
        return dict(op=op, B=B, NQ=sh.num_heads, NKV=sh.num_kv_heads, D=rng.choice([64, 128]), S=_log_int(rng, 64, 8192))
    if op == "attn":
        sh = SHAPES[model]
        S = _log_int(rng, 64, 8192)
        return dict(op=op, B=B, H=sh.num_heads, NKV=sh.num_kv_heads, D=rng.choice([64, 128]), S=S, min_len=rng.choice([0, max(1, S // 8)]))
    if op == "ffn":
        return dict(op=op, model=model, B=B)
    if op == "layer":
        return dict(op=op, model=model, B=B, S=_log_int(rng, 64, 8192))
    B = _log_int(rng, 1, 32)
    kind = rng.choice(["uniform", "ragged", "paged"])
    page = rng.choice([64, 128, 256]) if kind == "paged" else 0
    S = _log_int(rng, 64, 2048)
    if page:
        S = max(1, round(S / page)) * page
    return dict(op=op, model=model, B=B, S=S, layers=rng.randint(2, 6), ragged=kind != "uniform", page=page)


# ------------------------------------------------------------------- inputs ---
def _normal(g, *shape, std=1.0, mean=0.0, dtype=BF16):
    t = torch.randn(*shape, generator=g, device="cuda", dtype=dtype)
    if std != 1.0:
        t.mul_(std)
    if mean:
        t.add_(mean)
    return t


def _lengths(case, seed, low):
    """Per-row lengths in [low, S]: a property of the batch, drawn from the seed."""
    g = torch.Generator().manual_seed(seed)
    return torch.randint(low, case["S"] + 1, (case["B"],), generator=g).tolist()


def _weights(g, sh):
    H, I = sh.hidden, sh.inter
    return [_normal(g, n, k, std=0.02) for n, k in ((sh.q_rows + 2 * sh.kv_rows, H), (H, sh.q_rows), (2 * I, H), (H, I))]


def prepare(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    op = case["op"]
    if op == "gemv":
        N, K = case["N"], case["K"]
        y = torch.empty(N, device="cuda", dtype=BF16)
        return dict(op=op, fn=ez.GemvOp(N, K, backend="cuda"), args=(_normal(g, K), _normal(g, N, K, std=0.02), y), out=y)
    if op == "rmsnorm":
        rows, dim = case["rows"], case["dim"]
        if case["dtype"] == "bf16":
            X, w = _normal(g, rows, dim), _normal(g, dim, std=0.1, mean=1.0)
            out = torch.empty_like(X)
            return dict(op=op, fn=ez.RmsNormOp(rows, dim, backend="cuda", dtype=BF16, with_weight=True), args=(X, w, out), out=out)
        X = _normal(g, rows, dim, dtype=torch.float32)
        out = torch.empty_like(X)
        return dict(op=op, fn=ez.RmsNormOp(rows, dim, backend="cuda"), args=(X, out), out=out)
    if op == "qk_rope":
        B, NQ, NKV, D, S = (case[k] for k in ("B", "NQ", "NKV", "D", "S"))
        positions = [n - 1 for n in _lengths(case, seed, 1)]
        fn = ez.FusedQkNormRopeOp(B, NQ, D, S, positions, backend="cuda", num_kv_heads=NKV)
        cos, sin = (t.cuda() for t in wl.rope_tables(S, D))
        Kc, Vc = _normal(g, B, NKV, S, D), _normal(g, B, NKV, S, D)
        args = (_normal(g, B, NQ, D), _normal(g, B, NKV, D), _normal(g, B, NKV, D), _normal(g, D, std=0.1, mean=1.0),
                _normal(g, D, std=0.1, mean=1.0), cos, sin, Kc, Vc)
        return dict(op=op, fn=fn, args=args, caches=(Kc, Vc))
    if op == "attn":
        B, H, NKV, D, S = (case[k] for k in ("B", "H", "NKV", "D", "S"))
        lens = _lengths(case, seed, case["min_len"]) if case["min_len"] else None
        fn = ez.AttnDecodeOp(B, H, S, D, backend="cuda", num_kv_heads=NKV, seq_lens=lens)
        return dict(op=op, fn=fn, args=(_normal(g, B, H, 1, D), _normal(g, B, NKV, S, D), _normal(g, B, NKV, S, D)))
    sh, B = SHAPES[case["model"]], case["B"]
    H, I, D, NKV = sh.hidden, sh.inter, sh.head_dim, sh.num_kv_heads
    if op == "ffn":
        fn = ez.FusedOProjFfnOp(B, H, I, sh.num_heads, D, backend="cuda")
        args = (_normal(g, B, sh.q_rows), _normal(g, B, H), _normal(g, H, sh.q_rows, std=0.02), _normal(g, H, std=0.1, mean=1.0),
                _normal(g, I, H, std=0.02), _normal(g, I, H, std=0.02), _normal(g, H, I, std=0.02))
        return dict(op=op, fn=fn, args=args)
    S = case["S"]
    if op == "layer":
        fn = ez.Qwen3DenseDecodeOp(B, S, H, I, sh.num_heads, D, backend="cuda", num_kv_heads=NKV)
        Kc, Vc = _normal(g, B, NKV, S, D), _normal(g, B, NKV, S, D)
        return dict(op=op, fn=fn, args=(_normal(g, B, H), Kc, Vc, *_weights(g, sh)), caches=(Kc, Vc))
    # stack: the handle a decode loop keeps, and this step's hidden states, lengths and (paged) page table
    kernel = ez.get_kernel("qwen3_decode_stack", "cuda")(B, S, H, I, sh.num_heads, D, case["layers"], num_kv_heads=NKV)
    page = case["page"]
    cache = (B * S // page + 3, NKV, page, D) if page else (B, NKV, S, D)
    layers = []
    for _ in range(case["layers"]):
        Wqkv, Wo, Wgu, Wd = _weights(g, sh)
        layer = dict(K_cache=_normal(g, *cache), V_cache=_normal(g, *cache), Wqkv=Wqkv, Wo=Wo, Wgu=Wgu, Wd=Wd)
        for key, n in (("input_norm_w", H), ("post_norm_w", H), ("q_norm_w", D), ("k_norm_w", D)):
            layer[key] = _normal(g, n, std=0.1, mean=1.0)
        layers.append(layer)
    cos, sin = (t.cuda() for t in wl.rope_tables(S, D))
    kw = {}
    if case["ragged"]:
        kw["seq_lens"] = torch.tensor(_lengths(case, seed, max(1, S // 8)), dtype=torch.int32, device="cuda")
    if page:
        order = torch.randperm(cache[0], generator=torch.Generator().manual_seed(seed))[: B * S // page]
        kw["page_table"], kw["page_size"] = order.view(B, S // page).to(torch.int32).cuda(), page
    caches = tuple(t for L in layers for t in (L["K_cache"], L["V_cache"]))
    return dict(op=op, fn=kernel, args=(_normal(g, B, H), layers, cos, sin), kw=kw, caches=caches)


# --------------------------------------------------------------------- pass ---
def run(state):
    """One call.  Results are what the operator returns or writes: outputs and updated caches."""
    out = state["fn"](*state["args"], **state.get("kw", {}))
    if "out" in state:
        return state["out"]
    return (out, *state["caches"]) if "caches" in state else out


# --------------------------------------------------------------------- cost ---
def _mean_len(case, low):
    return (low + case["S"]) / 2 if low else case["S"]


def work(case):
    """Weights, valid keys and values, activations: each read or written once, two bytes an element (four in fp32)."""
    op = case["op"]
    if op == "gemv":
        N, K = case["N"], case["K"]
        return dict(bytes=2 * (N * K + N + K), flops=2 * N * K)
    if op == "rmsnorm":
        rows, dim, size = case["rows"], case["dim"], 2 if case["dtype"] == "bf16" else 4
        return dict(bytes=size * (2 * rows * dim + (dim if size == 2 else 0)), flops=4 * rows * dim)
    if op == "qk_rope":
        B, NQ, NKV, D = (case[k] for k in ("B", "NQ", "NKV", "D"))
        # q, k, v in; q, k out; k, v into the cache; one cos and one sin row per token
        return dict(bytes=2 * D * B * (2 * NQ + 5 * NKV + 2) + 4 * D + 4 * B, flops=10 * B * (NQ + NKV) * D)
    if op == "attn":
        B, H, NKV, D = (case[k] for k in ("B", "H", "NKV", "D"))
        n = B * _mean_len(case, case["min_len"])
        return dict(bytes=2 * D * (2 * n * NKV + 2 * B * H), flops=4 * n * H * D)
    sh, B = SHAPES[case["model"]], case["B"]
    H, Q = sh.hidden, sh.q_rows
    if op == "ffn":
        elems = H * Q + 3 * sh.inter * H
        return dict(bytes=2 * (elems + B * (Q + 2 * H) + H), flops=2 * B * elems)
    S = case["S"]
    n = B * (_mean_len(case, max(1, S // 8)) if case.get("ragged") else S)
    elems = sh.weight_bytes() // 2
    layer_bytes = 2 * elems + 4 * n * sh.kv_rows
    layers = case.get("layers", 1)
    return dict(bytes=layers * layer_bytes + 4 * B * H, flops=layers * (2 * B * elems + 4 * n * Q))


# Relative error and largest difference that another order of the sums brings, about four times what was measured
# between this path and itself with other splits and kernels (measured: attn 2.0e-3 / 7.8e-3, layer 3.6e-3 / 1.6e-2).
# Single projections, norms and rotations round once: a few values land on the other side of a bf16 rounding.
TOLERANCE = dict(
    gemv=dict(rel=1e-3, max=2e-2),
    rmsnorm=dict(rel=1e-3, max=2e-2),
    qk_rope=dict(rel=1e-3, max=2e-2),
    attn=dict(rel=8e-3, max=4e-2),
    ffn=dict(rel=8e-3, max=8e-2),
    layer=dict(rel=1.4e-2, max=8e-2),
)


def tolerance(case):
    if case["op"] == "rmsnorm" and case["dtype"] == "fp32":
        return dict(rel=1e-6)
    if case["op"] == "stack":
        # rounding differences add up along the residual stream: 4.0e-3 / 2.1e-2 after two layers, 1.2e-2 / 5.3e-2 after
        # eight, 1.6e-2 / 7.6e-2 after 28
        return dict(rel=1.6e-2, max=1e-1) if case["layers"] <= 2 else dict(rel=3e-2, max=3e-1)
    return TOLERANCE[case["op"]]


# -------------------------------------------------------------------- exact ---
def _norm64(x, weight=None):
    y = x * torch.rsqrt(x.square().mean(-1, keepdim=True) + 1e-6)
    return y if weight is None else y * weight.double()


def _rotate64(x, cos, sin):
    """x [B, heads, D], tables [B, D]: the two halves of a head are the rotated pairs."""
    a, b = x.chunk(2, -1)
    return x * cos.double()[:, None] + torch.cat([-b, a], -1) * sin.double()[:, None]


def _attend64(q, K, V, lens):
    """q [B, H, D]; K(b) and V(b) give a row's [NKV, S, D]; the first lens[b] keys count."""
    rows = []
    for b, n in enumerate(lens):
        k, v = K(b)[:, :n].double(), V(b)[:, :n].double()
        p = (q[b].view(k.shape[0], -1, k.shape[2]) @ k.transpose(1, 2) * k.shape[2] ** -0.5).softmax(-1)
        rows.append((p @ v).reshape(q.shape[1], -1))
    return torch.stack(rows)


def _swiglu64(x2, weight, Wg, Wu, Wd):
    xn = _norm64(x2, weight)
    return x2 + (torch.nn.functional.silu(xn @ Wg.double().T) * (xn @ Wu.double().T)) @ Wd.double().T


def _layer64(x, L, sh, lens, cos=None, sin=None, pages=None):
    """One layer in 64 bits; returns its output and the caches as they stand afterwards."""
    B, D, NKV = x.shape[0], sh.head_dim, sh.num_kv_heads
    qkv = _norm64(x, L.get("input_norm_w")) @ L["Wqkv"].double().T
    q, k, v = (t.reshape(B, -1, D) for t in qkv.split([sh.q_rows, sh.kv_rows, sh.kv_rows], -1))
    q, k = _norm64(q, L.get("q_norm_w")), _norm64(k, L.get("k_norm_w"))
    if cos is not None:
        at = torch.tensor(lens, device=x.device) - 1
        q, k = _rotate64(q, cos[at], sin[at]), _rotate64(k, cos[at], sin[at])
    Kc, Vc = L["K_cache"].double(), L["V_cache"].double()
    if pages is None:
        row = lambda t: lambda b: t[b]  # noqa: E731
    else:
        row = lambda t: lambda b: t[pages[b].long()].transpose(0, 1).reshape(NKV, -1, D)  # noqa: E731
    for b, n in enumerate(lens):
        slot = (b, n - 1) if pages is None else (int(pages[b, (n - 1) // Kc.shape[2]]), (n - 1) % Kc.shape[2])
        Kc[slot[0], :, slot[1]], Vc[slot[0], :, slot[1]] = k[b], v[b]
    x2 = x + _attend64(q, row(Kc), row(Vc), lens).reshape(B, -1) @ L["Wo"].double().T
    Wg, Wu = L["Wgu"].chunk(2)
    return _swiglu64(x2, L.get("post_norm_w"), Wg, Wu, L["Wd"]), Kc, Vc


def exact(case, seed):
    """What ``run`` returns for these inputs, computed by torch in 64 bits with no rounding in between."""
    state = prepare(case, seed)
    args, op = state["args"], case["op"]
    if op == "gemv":
        return args[1].double() @ args[0].double()
    if op == "rmsnorm":
        return _norm64(args[0].double(), args[1] if case["dtype"] == "bf16" else None)
    if op == "qk_rope":
        q, k, v, qw, kw, cos, sin, Kc, Vc = args
        at = [n - 1 for n in _lengths(case, seed, 1)]
        q, k = (_rotate64(_norm64(t.double(), w), cos[at], sin[at]) for t, w in ((q, qw), (k, kw)))
        Kc, Vc = Kc.double(), Vc.double()
        for b, slot in enumerate(at):
            Kc[b, :, slot], Vc[b, :, slot] = k[b], v[b].double()
        return (q, k), Kc, Vc
    if op == "attn":
        Q, K, V = args
        lens = _lengths(case, seed, case["min_len"]) if case["min_len"] else [case["S"]] * case["B"]
        return _attend64(Q[:, :, 0].double(), lambda b: K[b], lambda b: V[b], lens)[:, :, None]
    if op == "ffn":
        attn, residual, Wo, weight, Wg, Wu, Wd = args
        return _swiglu64(residual.double() + attn.double() @ Wo.double().T, weight, Wg, Wu, Wd)
    sh, B, S = SHAPES[case["model"]], case["B"], case["S"]
    if op == "layer":
        names = ("K_cache", "V_cache", "Wqkv", "Wo", "Wgu", "Wd")
        return _layer64(args[0].double(), dict(zip(names, args[1:])), sh, [S] * B)
    hidden, layers, cos, sin = args
    lens = _lengths(case, seed, max(1, S // 8)) if case["ragged"] else [S] * B
    x, caches = hidden.double(), []
    for L in layers:
        x, *kv = _layer64(x, L, sh, lens, cos, sin, state["kw"].get("page_table"))
        caches += kv
    return (x, *caches)
