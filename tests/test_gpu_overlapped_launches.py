"""Kernels whose launch overlaps the end of the kernel in front of them: results, and the room that they leave to others.

No kernel here waits for another that runs beside it: a wait that is meant to last ends at its own limit."""
import ctypes
import time

import pytest
import torch

from nixl_b200.ops import _lib, grouped_gemm_fp8, quantize_weights
from nixl_b200.parallel import Buffer, per_token_cast_to_fp8

pytestmark = pytest.mark.gpu


def _routing(tokens, hidden, experts, topk, seed):
    dev = torch.device("cuda:0")
    g = torch.Generator(device=dev).manual_seed(seed)
    x = torch.randn(tokens, hidden, device=dev, dtype=torch.bfloat16, generator=g)
    w, idx = torch.topk(torch.softmax(torch.randn(tokens, experts, device=dev, generator=g), -1), topk, -1)
    return x, idx.contiguous(), w.float().contiguous()


def _gemm(groups, n, k, rows_each, seed, **kw):
    """A grouped GEMM that can be launched again and again into the same output."""
    dev = torch.device("cuda:0")
    g = torch.Generator(device=dev).manual_seed(seed)
    a, sa = per_token_cast_to_fp8(torch.randn(groups * rows_each, k, device=dev, generator=g).to(torch.bfloat16))
    wq, sw = quantize_weights(torch.randn(groups, n, k, device=dev, generator=g) * 0.05)
    rs = torch.arange(groups, device=dev, dtype=torch.int32) * rows_each
    rc = torch.full_like(rs, rows_each)
    out = torch.empty(groups * rows_each, n, device=dev, dtype=torch.bfloat16)
    status = torch.zeros(1, dtype=torch.int32, device=dev)
    return lambda: grouped_gemm_fp8(a, sa, wq, sw, rs, rc, out=out, status=status, **kw)


@pytest.mark.parametrize("rows_each", [8, 128])  # both forms of the single-CTA kernel
def test_receive_that_waits_leaves_the_sms_to_other_streams(rows_each):
    """A receive whose flags are not up waits; the GEMM behind it in the stream must not sit on the other SMs meanwhile."""
    T, H, E, K = 64, 512, 8, 2
    dev = torch.device("cuda:0")
    b = Buffer(0, 1, E, H, T, K, device=dev, low_latency_mode=True, timeout_ms=400)
    b.connect_ranks()
    b.set_num_sms(4)
    behind, elsewhere = _gemm(8, 4096, 512, rows_each, 1), _gemm(8, 1024, 512, rows_each, 2, grid=64)
    x, idx, _ = _routing(T, H, E, K, 3)
    _, _, h, _, hook = b.low_latency_dispatch(x, idx, use_fp8=False, return_recv_hook=True)
    hook()
    behind()
    want = elsewhere().clone()  # (everything has been launched once: nothing is loaded later)
    p = b._disp_cache[(h.parity, False, h.rows_per_expert, False)][0]
    flags = b._region(h.parity, "off_disp_flag", E * 8).view(torch.int64)
    flags[1] = 0  # one expert's rows "not yet there"
    waits, other = torch.cuda.Stream(dev), torch.cuda.Stream(dev)
    received = torch.cuda.Event()
    torch.cuda.synchronize()
    with torch.cuda.stream(waits):
        p.phases = 2
        _lib.check(b._dispatch_fn(ctypes.byref(p), _lib.raw_stream(dev)), "dispatch")
        received.record()
        behind()
    time.sleep(0.05)
    with torch.cuda.stream(other):
        got = elsewhere()
        done = other.record_event()
    done.synchronize()
    assert not received.query(), "the GEMM on the other stream ran only when the receive had given up"
    torch.cuda.synchronize()
    assert b.status & 1 and torch.equal(got, want)
    b.destroy()
