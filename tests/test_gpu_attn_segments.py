"""Attention inside a stack of layers over rows of different lengths: a CTA that takes several segments in turn (norm weights,
rotary row and the new token's key and value per segment, the next segment's tiles requested while one is merged), over
contiguous and paged caches, and a captured graph replayed after the lengths have changed on the device."""

import random

import pytest
import torch

from ezops_b200 import _lib
from ezops_b200 import workloads as wl

pytestmark = pytest.mark.gpu

NH, NKV, LAYERS = 16, 8, 2
# (batch, longest row, shortest row, head_dim, page): what the lengths lead to is said beside it
CASES = [
    (32, 2048, 64, 128, 0),  # ranges: a CTA ends one group and begins the next
    (32, 2048, 64, 128, 256),
    (48, 1536, 1, 64, 64),
    (64, 512, 1, 128, 0),  # whole groups, or one CTA per group
    (64, 256, 1, 64, 128),
    (13, 1024, 128, 128, 64),  # pieces
]


def _lengths(B, S, low, seed):
    rng = random.Random(seed)
    lens = [rng.randint(low, S) for _ in range(B)]
    lens[0], lens[-1] = S, low
    return lens


def _inputs(B, S, D, page, seed=0):
    """Layers whose output is their input plus the attention's result: the output projection is the identity, the FFN's
    last projection zero.  The input is small beside that result, so its rounding does not hide an error in it."""
    H, I = NH * D, 256
    g = torch.Generator(device="cuda").manual_seed(seed + B + S)
    rand = lambda *s, std=1.0, mean=0.0: (torch.randn(*s, generator=g, device="cuda") * std + mean).bfloat16()  # noqa: E731
    layers = []
    for _ in range(LAYERS):
        layers.append(dict(
            K_cache=rand(B, NKV, S, D), V_cache=rand(B, NKV, S, D), Wqkv=rand((NH + 2 * NKV) * D, H, std=0.02),
            Wo=torch.eye(H, device="cuda").bfloat16(), Wgu=rand(2 * I, H, std=0.02), Wd=torch.zeros(H, I, device="cuda").bfloat16(),
            input_norm_w=rand(H, std=0.1, mean=1.0), post_norm_w=rand(H, std=0.1, mean=1.0),
            q_norm_w=rand(D, std=0.1, mean=1.0), k_norm_w=rand(D, std=0.1, mean=1.0)))
    cos, sin = (t.cuda() for t in wl.rope_tables(S, D))
    table = None
    if page:
        per_row = S // page
        perm = torch.randperm(B * per_row + 3, generator=torch.Generator().manual_seed(B))[: B * per_row].view(B, per_row)
        table = perm.to(torch.int32).cuda()
    return rand(B, H, std=0.01), layers, cos, sin, table


def _paged(cache, table, page):
    B, heads, S, D = cache.shape
    pool = torch.randn(table.numel() + 3, heads, page, D, device="cuda").bfloat16()
    pool[table.flatten().long()] = cache.view(B, heads, S // page, page, D).transpose(1, 2).reshape(-1, heads, page, D)
    return pool


def _contiguous(pool, table, page):
    B, n = table.shape
    return pool[table.flatten().long()].view(B, n, pool.shape[1], page, -1).transpose(1, 2).reshape(B, pool.shape[1], n * page, -1)


def _expected(hidden, layers, cos, sin, lens):
    """In 64 bits: hidden states behind the last layer and, per layer, the token's new key and value."""
    norm = lambda x, w: x * torch.rsqrt(x.square().mean(-1, keepdim=True) + 1e-6) * w.double()  # noqa: E731
    B, D = hidden.shape[0], cos.shape[1]
    x, new = hidden.double(), []
    at = torch.tensor(lens, device="cuda") - 1
    c, s = cos[at].double()[:, None], sin[at].double()[:, None]

    def rotate(t):
        a, b = t.chunk(2, -1)
        return t * c + torch.cat([-b, a], -1) * s

    for L in layers:
        qkv = norm(x, L["input_norm_w"]) @ L["Wqkv"].double().T
        q, k, v = (t.reshape(B, -1, D) for t in qkv.split([NH * D, NKV * D, NKV * D], -1))
        q, k = rotate(norm(q, L["q_norm_w"])), rotate(norm(k, L["k_norm_w"]))
        out = []
        for b, n in enumerate(lens):
            K = torch.cat([L["K_cache"][b, :, : n - 1].double(), k[b][:, None]], 1)
            V = torch.cat([L["V_cache"][b, :, : n - 1].double(), v[b][:, None]], 1)
            p = (q[b].view(NKV, -1, D) @ K.transpose(1, 2) * D**-0.5).softmax(-1)
            out.append((p @ V).reshape(-1))
        x = x + torch.stack(out)
        new.append((k, v))
    return x, new


def _stack(B, S, D):
    import ezops_b200 as ez

    return ez.get_kernel("qwen3_decode_stack", "cuda")(B, S, NH * D, 256, NH, D, LAYERS, num_kv_heads=NKV)


@pytest.mark.parametrize("B,S,low,D,page", CASES)
def test_stack_over_rows_of_different_lengths(B, S, low, D, page):
    """Row by row against 64 bits.  Two layers, in each of which the normalised row, q, k, v, the probabilities, the result
    and the sum with the residual are rounded to bf16 (2**-8 at most each, uniformly spread: 2**-9.8 on average): 2e-2 of
    a row's norm is above seven roundings that all add up and below what one missing tile of 64 keys in 2048 changes
    (18 %)."""
    hidden, layers, cos, sin, table = _inputs(B, S, D, page)
    lens = _lengths(B, S, low, B * S)
    want, new = _expected(hidden, layers, cos, sin, lens)
    before = [(L["K_cache"].clone(), L["V_cache"].clone()) for L in layers]
    kw = dict(seq_lens=torch.tensor(lens, dtype=torch.int32, device="cuda"))
    if page:
        layers = [{**L, "K_cache": _paged(L["K_cache"], table, page), "V_cache": _paged(L["V_cache"], table, page)} for L in layers]
        kw.update(page_table=table, page_size=page)
    kernel = _stack(B, S, D)
    got = kernel(hidden, layers, cos, sin, **kw)
    assert _lib.device_status() == 0
    off = (got.double() - want).norm(dim=-1) / want.norm(dim=-1)
    assert off.max().item() < 2e-2, (off.argmax().item(), off.max().item())
    rows, slots = torch.arange(B, device="cuda"), torch.tensor(lens, device="cuda") - 1
    for L, (K0, V0), (k, v) in zip(layers, before, new):
        K, V = (_contiguous(L[n], table, page) if page else L[n] for n in ("K_cache", "V_cache"))
        for cache, old, token in ((K, K0, k), (V, V0, v)):
            assert ((cache[rows, :, slots].double() - token).norm(dim=(1, 2)) / token.norm(dim=(1, 2))).max().item() < 2e-2
            cache = cache.clone()
            cache[rows, :, slots] = old[rows, :, slots]
            assert torch.equal(cache, old)  # nothing but the token's slot was written
    assert torch.equal(kernel(hidden, layers, cos, sin, **kw), got)  # the written slot is the one it is replaced by


@pytest.mark.parametrize("B,S,D,page", [(32, 2048, 128, 256), (48, 1024, 64, 0)])
def test_replay_follows_the_lengths(B, S, D, page):
    """One captured call, replayed over lengths that lead to every form of the schedule and written directly in front of
    it: the bits of an eager call with the same lengths."""
    hidden, layers, cos, sin, table = _inputs(B, S, D, page)
    if page:
        layers = [{**L, "K_cache": _paged(L["K_cache"], table, page), "V_cache": _paged(L["V_cache"], table, page)} for L in layers]
    before = [(L["K_cache"].clone(), L["V_cache"].clone()) for L in layers]
    many = [_lengths(B, S, 1, 1), [1] * B, [S] * B, _lengths(B, 200, 1, 2), _lengths(B, S, S // 2, 3), [S] + [40] * (B - 1)]
    many = [torch.tensor(n, dtype=torch.int32, device="cuda") for n in many]
    lens = many[0].clone()
    kw = dict(seq_lens=lens, **(dict(page_table=table, page_size=page) if page else {}))
    kernel, out = _stack(B, S, D), torch.empty_like(hidden)

    def restore():
        for L, (K0, V0) in zip(layers, before):
            L["K_cache"].copy_(K0)
            L["V_cache"].copy_(V0)

    want = []
    for n in many:
        restore()
        lens.copy_(n)
        want.append((kernel(hidden, layers, cos, sin, **kw).clone(), layers[-1]["K_cache"].clone()))
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        kernel(hidden, layers, cos, sin, out=out, **kw)
    for order in (range(len(many)), reversed(range(len(many)))):
        for i in order:
            restore()
            lens.copy_(many[i])
            graph.replay()
            assert torch.equal(out, want[i][0]) and torch.equal(layers[-1]["K_cache"], want[i][1]), i
    assert _lib.device_status() == 0
