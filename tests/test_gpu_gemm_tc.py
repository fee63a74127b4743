"""The tensor-core projection kernel (csrc/gemm_tc.cu) at the edges of its plan: tiles of 8 to 128 rows, clusters of 1 to
8 CTAs, several rounds of tiles per cluster, K that ends inside a 64-element block, batches that fill a column tile or
leave most of it empty."""

import pytest
import torch

from ezops_b200 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B", [9, 16, 17, 32, 33, 64])
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
