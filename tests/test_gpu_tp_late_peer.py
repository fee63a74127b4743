"""The budget for a peer's partial sums is EZB_TUNE_TP_WAIT_LIMIT_MS, whatever else waits meanwhile: the waits inside a
kernel (about one second) neither run while the kernel in front still waits for its peers nor end a kernel whose own gather
does."""

import ctypes

import pytest
import torch

from ezops_b200 import _lib
from ezops_b200 import workloads as wl

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,mega", [(1, 1), (1, 0), (2, 1), (16, 1)])
def test_late_peer_is_waited_for_as_long_as_the_limit_says(B, mega):
    """A world of two whose second rank nobody plays, both communication buffers on this GPU, budget 1.5 s: the call
    returns after that time and not after the second that other waits have, the status word names the exchange (0x201),
    nothing is published.  The single-kernel layer, the chained kernels of one row, and the tensor-core form."""
    lib = _lib.load()
    sh, S = wl.QWEN3_0_6B, 200
    hidden, Kc, Vc, Wqkv, Wo, Wgu, Wd = (t.cuda() for t in wl.decode_layer_inputs(sh, B, S))
    bufs = [ctypes.c_void_p(), ctypes.c_void_p()]
    for b in bufs:
        _lib.check(lib.ezb_tp_comm_alloc(lib.ezb_tp_comm_bytes(B, sh.hidden), ctypes.byref(b)))
    ws = torch.zeros(lib.ezb_qwen3_decode_layer_workspace_bytes(B, S, sh.hidden, sh.inter, sh.num_heads, sh.num_kv_heads, sh.head_dim),
                     dtype=torch.uint8, device="cuda")
    out = torch.full_like(hidden, 7.0)
    bases = (ctypes.c_void_p * 2)(*[b.value for b in bufs])

    def call():
        _lib.check(lib.ezb_qwen3_decode_layer_tp_fused(
            hidden.data_ptr(), Kc.data_ptr(), Vc.data_ptr(), Wqkv.data_ptr(), Wo.data_ptr(), Wgu.data_ptr(), Wd.data_ptr(),
            out.data_ptr(), ws.data_ptr(), ws.numel(), bases, 2, 0, B, S, sh.hidden, sh.inter, sh.num_heads,
            sh.num_kv_heads, sh.head_dim, 1e-6, torch.cuda.current_stream().cuda_stream))

    t0, t1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    try:
        _lib.set_tuning(tp_wait_limit_ms=1500, mega=mega)
        t0.record()
        call()
        t1.record()
        torch.cuda.synchronize()
        word = ctypes.c_uint(0)
        assert lib.ezb_device_status(ctypes.byref(word), 0) == _lib.EZB_ERR_DEVICE_FAULT and word.value == 0x201
        # the limit is in cycles at 2 GHz, the clock is 1.965 GHz at most
        assert 1490.0 < t0.elapsed_time(t1) < 4000.0
        assert torch.equal(out, torch.full_like(out, 7.0)), "a rank that gave up must not publish a result"
        # while the fault stands: silent, and quick
        t0.record()
        call()
        t1.record()
        torch.cuda.synchronize()
        assert t0.elapsed_time(t1) < 50.0 and torch.equal(out, torch.full_like(out, 7.0))
        assert _lib.device_status() == 0x201  # reads and clears
    finally:
        _lib.set_tuning(tp_wait_limit_ms=5000, mega=1)
        torch.cuda.synchronize()
        _lib.device_status()
        for b in bufs:
            _lib.check(lib.ezb_tp_comm_free(b))
