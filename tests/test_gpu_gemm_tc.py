"""The tensor-core projection kernel (csrc/gemm_tc.cu) at the edges of its plan: tiles of 8 to 128 rows, clusters of 1 to
8 CTAs, several rounds of tiles per cluster, K that ends inside a 64-element block, batches that fill a column tile or
leave most of it empty."""

import pytest
import torch

from ezops_b200 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B", [2, 3, 5, 8, 9, 16, 17, 32, 33, 64])
@pytest.mark.parametrize("N,K", [(1, 16), (8, 64), (9, 80), (130, 80), (1024, 2048), (1023, 4112), (4097, 64), (10240, 144), (40001, 256)])
def test_batched_projection(B, N, K):
    """Against the fp32 product: bf16 products are exact in fp32, so what differs is the order of K fp32 additions
    (relative to the sum of magnitudes at most K * 2**-24, and far less in practice) and the rounding of the result to
    bf16 (8 significant bits: half a unit in the last place is at most 2**-8 of the value)."""
    lib = _lib.load()
    g = torch.Generator().manual_seed(1000 * B + N + K)
    X = torch.randn(B, K, generator=g).bfloat16().cuda()
    W = (torch.randn(N, K, generator=g) * 0.02).bfloat16().cuda()
    Y = torch.full((B, N), float("nan"), dtype=torch.bfloat16, device="cuda")
    ws = torch.zeros(lib.ezb_gemv_workspace_bytes(B, N, K), dtype=torch.uint8, device="cuda")
    call = lambda: _lib.check(lib.ezb_gemv_batched_bf16(X.data_ptr(), W.data_ptr(), Y.data_ptr(), ws.data_ptr(), ws.numel(), B, N, K,  # noqa: E731
                                                        torch.cuda.current_stream().cuda_stream))
    call()
    assert _lib.device_status() == 0
    want = X.double() @ W.double().T
    bound = 2.0**-8 * want.abs() + K * 2.0**-24 * (X.double().abs() @ W.double().abs().T)
    assert ((Y.double() - want).abs() <= bound * 1.01).all()
    first = Y.clone()
    call()
    assert torch.equal(first, Y)  # fixed order of the sums


@pytest.mark.parametrize("B", [2, 8, 9, 32, 64])
@pytest.mark.parametrize("H,I,NH", [(64, 16, 1), (1040, 1048 * 2, 3), (2048, 6144, 16)])
def test_projection_epilogues(B, H, I, NH):
    """Residual and SwiGLU epilogues through the output projection + FFN operator, in 64 bits from the same rounding
    points: each of the four projections and the norm rounds to bf16 once (2**-8 at most), and 1e-2 of the norm is the operator's own bound."""
    import ezops_b200 as ez

    D = 64
    g = torch.Generator().manual_seed(B + H)
    r = lambda *s, std=1.0, mean=0.0: (torch.randn(*s, generator=g) * std + mean).bfloat16().cuda()  # noqa: E731
    op = ez.FusedOProjFfnOp(B, H, I, NH, D, backend="cuda")
    attn, residual, Wo, w = r(B, NH * D), r(B, H), r(H, NH * D, std=0.02), r(H, std=0.1, mean=1.0)
    Wg, Wu, Wd = r(I, H, std=0.02), r(I, H, std=0.02), r(H, I, std=0.02)
    out = op(attn, residual, Wo, w, Wg, Wu, Wd)
    assert _lib.device_status() == 0
    x2 = residual.double() + attn.double() @ Wo.double().T
    xn = x2 * torch.rsqrt(x2.square().mean(-1, keepdim=True) + 1e-6) * w.double()
    want = x2 + (torch.nn.functional.silu(xn @ Wg.double().T) * (xn @ Wu.double().T)) @ Wd.double().T
    assert ((out.double() - want).norm() / want.norm()).item() < 1e-2
    assert torch.equal(out, op(attn, residual, Wo, w, Wg, Wu, Wd))


# ------------------------------------------------------------------------------------ epilogues, value by value ---
STEP = 2.0**-8  # a rounding to bf16 changes a value by at most this share of it; 2**-8.8 is its standard deviation at most
BATCHES = [2, 3, 5, 8, 9, 17, 32, 64]
SIZES = [(64, 16, 1), (1040, 2096, 3), (2048, 6144, 16)]  # H, I, heads of 64


def _ffn(B, H, I, NH, seed):
    import ezops_b200 as ez

    g = torch.Generator().manual_seed(seed)
    rand = lambda *s, std=1.0, mean=0.0: (torch.randn(*s, generator=g) * std + mean).bfloat16().cuda()  # noqa: E731
    return ez.FusedOProjFfnOp(B, H, I, NH, 64, backend="cuda"), rand


@pytest.mark.parametrize("B", BATCHES)
@pytest.mark.parametrize("H,I,NH", SIZES)
def test_residual_epilogue_value_by_value(B, H, I, NH):
    """The FFN's last projection is zero, so the operator returns residual + attn Wo^T: every value of it within the
    rounding of the product, that of the sum, and Q fp32 additions (at most 2**-24 of the magnitudes each)."""
    op, rand = _ffn(B, H, I, NH, B + H)
    Q = NH * 64
    attn, residual, Wo, w = rand(B, Q), rand(B, H, std=0.5), rand(H, Q, std=Q**-0.5), rand(H, std=0.1, mean=1.0)
    Wg, Wu, Wd = rand(I, H, std=0.02), rand(I, H, std=0.02), torch.zeros(H, I, device="cuda", dtype=torch.bfloat16)
    out = op(attn, residual, Wo, w, Wg, Wu, Wd)
    assert _lib.device_status() == 0
    prod = attn.double() @ Wo.double().T
    want = residual.double() + prod
    bound = STEP * (prod.abs() + want.abs()) + Q * 2.0**-24 * (attn.double().abs() @ Wo.double().abs().T)
    assert ((out.double() - want).abs() <= 1.01 * bound).all()


@pytest.mark.parametrize("B", BATCHES)
@pytest.mark.parametrize("H,I,NH", SIZES)
def test_swiglu_and_deferred_norm_value_by_value(B, H, I, NH):
    """The output projection is zero and the last projection picks one value of silu(gate) * up per output, so the
    operator returns residual + that value; shifted picks return every one of them.  gate and up are sums of products of
    rows rounded to bf16 once: independent errors, within eight standard deviations; then one rounding each, and one
    each for silu, the product and the sum.  silu has slope 1.1 at most."""
    op, rand = _ffn(B, H, I, NH, 7 * B + H)
    Q = NH * 64
    attn, residual, w = rand(B, Q), rand(B, H, std=0.0625), rand(H, std=0.1, mean=1.0)
    Wo = torch.zeros(H, Q, device="cuda", dtype=torch.bfloat16)
    Wg, Wu = rand(I, H, std=H**-0.5), rand(I, H, std=H**-0.5)
    x = residual.double()
    xn = x * torch.rsqrt(x.square().mean(-1, keepdim=True) + 1e-6) * w.double()

    def project(W):
        v = xn @ W.double().T
        return v, STEP * v.abs() + 8 * 2.0**-8.8 * (xn.square() @ W.double().square().T).sqrt()

    (gate, dg), (up, du) = project(Wg), project(Wu)
    s = torch.nn.functional.silu(gate)
    h = s * up
    ds = 1.1 * dg + STEP * s.abs()
    dh = (up.abs() + du) * ds + (s.abs() + ds) * du + STEP * h.abs()
    j = torch.arange(H, device="cuda")
    for first in range(0, I, H):
        pick = (j + first) % I
        Wd = torch.zeros(H, I, device="cuda", dtype=torch.bfloat16)
        Wd[j, pick] = 1.0
        out = op(attn, residual, Wo, w, Wg, Wu, Wd)
        want = x + h[:, pick]
        assert ((out.double() - want).abs() <= 1.01 * (dh[:, pick] + STEP * (want.abs() + dh[:, pick]))).all()
    assert _lib.device_status() == 0


@pytest.mark.parametrize("B", [2, 5, 8])
@pytest.mark.parametrize("N,K", [(1, 32), (8, 64), (130, 96), (1023, 4128), (4097, 64), (2048, 4096)])
def test_small_batch_kernel_without_the_tensor_cores(B, N, K):
    """What EZB_TUNE_TC = 0 selects for 2 to 8 rows (csrc/gemv_stream.cu); the bound of test_batched_projection."""
    try:
        _lib.set_tuning(tc=0)
        test_batched_projection(B, N, K)
    finally:
        _lib.set_tuning(tc=1)


@pytest.mark.parametrize("B,N,K,small", [
    (2, 2048, 8192, True),  # rows x K up to 16384, 2048 outputs
    (4, 2048, 4096, True),
    (3, 130, 1024, True),
    (4, 2048, 4128, False),  # past each edge
    (2, 2049, 1024, False),
    (5, 1024, 1024, False),
    (2, 1024, 80, False),  # K the small-batch kernel does not take
])
def test_which_kernel_a_small_batch_runs_on(B, N, K, small):
    """Both sides of the rule of ezb_gemv_batched_bf16: right values on each, and inside it the bits of the small-batch
    kernel (the tensor cores add in another order, which shows in a few of so many roundings)."""
    test_batched_projection(B, N, K)
    if not small:
        return
    lib = _lib.load()
    X, W = (torch.randn(n, K, device="cuda").bfloat16() for n in (B, N))
    ws = torch.zeros(lib.ezb_gemv_workspace_bytes(B, N, K), dtype=torch.uint8, device="cuda")
    got = []
    try:
        for tc in (1, 0):
            _lib.set_tuning(tc=tc)
            got.append(torch.empty(B, N, device="cuda", dtype=torch.bfloat16))
            _lib.check(lib.ezb_gemv_batched_bf16(X.data_ptr(), W.data_ptr(), got[-1].data_ptr(), ws.data_ptr(), ws.numel(), B, N, K,
                                                 torch.cuda.current_stream().cuda_stream))
    finally:
        _lib.set_tuning(tc=1)
    assert torch.equal(*got)
