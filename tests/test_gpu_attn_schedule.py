"""Attention over rows of different lengths: the balanced schedule of csrc/attn_decode.cu in each of its forms (pieces of
groups, whole groups, ranges across groups), the fixed grid it leaves to small batches and to more rows than it covers, and
the folds of few and of many parts."""

import random

import pytest
import torch

from ezops_b200 import _lib

pytestmark = pytest.mark.gpu

CASES = [
    (1, 8, 8, 200, 64, 1),  # one row, a few tiles
    (4, 16, 8, 640, 128, 0),  # empty rows among them
    (13, 16, 8, 1024, 128, 128),  # pieces
    (64, 32, 8, 100, 128, 1),  # whole groups
    (64, 16, 8, 300, 64, 0),
    (24, 32, 8, 3000, 128, 100),  # ranges
    (40, 8, 8, 4096, 64, 1),  # ranges, head_dim 64
    (128, 16, 8, 257, 128, 1),  # the most rows the schedule covers
    (129, 8, 8, 257, 128, 1),  # one more
    (2, 64, 2, 3000, 128, 10),  # two query tiles per kv head
    (101, 4, 1, 6000, 128, 1),  # one long row among short ones: its group has many parts
    (1, 16, 1, 8192, 128, 8192),  # more parts than the fast fold takes
]


@pytest.mark.parametrize("B,H,NKV,S,D,low", CASES)
def test_ragged_attention(B, H, NKV, S, D, low):
    """In 64 bits from the same inputs.  Probabilities are rounded to bf16 for the second product (2**-9 on average over
    many keys) and the result once (at most 2**-8): 6e-3 of the norm, the bound of the other attention tests."""
    rng = random.Random(B * S)
    lens = [rng.randint(low, S) for _ in range(B)]
    if (B, NKV) == (101, 1):
        lens = [rng.randint(1, 64) for _ in range(B)]
        lens[50] = S
    g = torch.Generator(device="cuda").manual_seed(B + S)
    rand = lambda *s: torch.randn(*s, generator=g, device="cuda", dtype=torch.bfloat16)  # noqa: E731
    Q, K, V = rand(B, H, 1, D), rand(B, NKV, S, D), rand(B, NKV, S, D)
    lens_dev = torch.tensor(lens, dtype=torch.int32, device="cuda")
    lib = _lib.load()
    ws = torch.zeros(lib.ezb_attn_decode_workspace_bytes(B, H, NKV, S, D), dtype=torch.uint8, device="cuda")
    outs = []
    for _ in range(2):
        out = torch.full_like(Q, float("nan"))
        _lib.check(lib.ezb_attn_decode(Q.data_ptr(), K.data_ptr(), V.data_ptr(), out.data_ptr(), ws.data_ptr(), ws.numel(), B, H, NKV, S, D,
                                       lens_dev.data_ptr(), torch.cuda.current_stream().cuda_stream))
        outs.append(out)
    assert _lib.device_status() == 0
    assert torch.equal(*outs)  # whichever CTA finishes a group, its parts are added in the same order
    for b, n in enumerate(lens):
        if n == 0:
            assert (outs[0][b] == 0).all()
            continue
        q, k, v = Q[b, :, 0].double().view(NKV, H // NKV, D), K[b, :, :n].double(), V[b, :, :n].double()
        want = ((q @ k.transpose(1, 2) * D**-0.5).softmax(-1) @ v).reshape(H, D)
        assert ((outs[0][b, :, 0].double() - want).norm() / want.norm()).item() < 6e-3, (b, n)
