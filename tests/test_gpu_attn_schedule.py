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
    (64, 32, 8, 100, 128, 1),  # one CTA per group
    (64, 16, 8, 300, 64, 0),
    (96, 32, 8, 300, 128, 1),  # whole groups
    (24, 32, 8, 3000, 128, 100),  # ranges
    (24, 8, 8, 4096, 64, 1),  # ranges, head_dim 64
    (40, 8, 8, 4096, 64, 1),  # fixed grid, head_dim 64
    (1, 32, 8, 8192, 64, 8000),  # few and short groups, head_dim 64: one wave of splits, more than the fast fold takes
    (5, 16, 16, 900, 64, 1),
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


def _ctas(B, H, NKV, S, D, lens):
    """CTAs that a call runs on: one trace record each."""
    Q, out = (torch.zeros(B, H, 1, D, device="cuda", dtype=torch.bfloat16) for _ in range(2))
    K, V = (torch.zeros(B, NKV, S, D, device="cuda", dtype=torch.bfloat16) for _ in range(2))
    lib = _lib.load()
    ws = torch.zeros(lib.ezb_attn_decode_workspace_bytes(B, H, NKV, S, D), dtype=torch.uint8, device="cuda")
    records = torch.zeros(4096 * 6, dtype=torch.int64, device="cuda")
    cursor = torch.zeros(1, dtype=torch.int32, device="cuda")
    try:
        _lib.check(lib.ezb_trace_enable(records.data_ptr(), cursor.data_ptr(), 4096))
        _lib.check(lib.ezb_attn_decode(Q.data_ptr(), K.data_ptr(), V.data_ptr(), out.data_ptr(), ws.data_ptr(), ws.numel(), B, H, NKV, S, D,
                                       None if lens is None else lens.data_ptr(), torch.cuda.current_stream().cuda_stream))
        torch.cuda.synchronize()
    finally:
        _lib.check(lib.ezb_trace_enable(None, None, 0))
    assert _lib.device_status() == 0
    return cursor.item()


@pytest.mark.parametrize("B,H,NKV,S,D,ctas", [
    (64, 32, 8, 100, 128, 64 * 8),  # a row is one split: one CTA per (row, kv head)
    (128, 32, 8, 384, 128, 128 * 8),  # more groups than the fixed grid cuts
    (64, 32, 8, 512, 64, 64 * 8 * 2),  # head_dim 64, many short groups: two splits each
    (1, 32, 8, 8192, 64, 8 * 43),  # head_dim 64, few and short groups: splits of 192 keys, one wave
    (4, 16, 8, 1024, 128, 4 * 8 * 8),  # the smallest splits of full rows fit one wave
    (32, 32, 8, 8192, 128, None),  # balanced: two CTAs per SM
    (11, 32, 8, 4096, 64, None),  # head_dim 64, few long groups: three
])
def test_which_shapes_are_balanced(B, H, NKV, S, D, ctas):
    """Which grid a batch of rows of different lengths runs on (trace records: one per CTA).  The balanced schedule is slower
    where the hardware hands out whole groups one by one, see launch_attn_instance."""
    if ctas is None:
        ctas = torch.cuda.get_device_properties(0).multi_processor_count * (2 if D == 128 else 3)
    rng = random.Random(B)
    lens = torch.tensor([rng.randint(S // 8, S) for _ in range(B)], dtype=torch.int32, device="cuda")
    assert _ctas(B, H, NKV, S, D, lens) == ctas


@pytest.mark.parametrize("D,per_sm", [(64, 3), (128, 2)])
@pytest.mark.parametrize("B,S", [(1, 8192), (5, 4096), (8, 8192), (16, 1024), (24, 2048), (32, 512)])
def test_rows_of_one_length_run_in_one_wave(B, S, D, per_sm):
    """No more CTAs than are resident together (160 registers a thread leave room for three at head_dim 64, the ring for two
    at 128): a second, partly filled wave costs a whole pass over a split."""
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    assert B * 8 <= _ctas(B, 32, 8, S, D, None) <= sms * per_sm
