"""A group of one rank, whose kernels take shorter ways: what they publish, leave alone and accept must be as for a larger group.

No kernel here waits for another that runs beside it: where one kernel consumes another's flags on a second stream, the host
lets the first one end before it launches the second."""
import pytest
import torch

from nixl_b200.ops import grouped_gemm_fp8, quantize_weights
from nixl_b200.parallel import Buffer

pytestmark = pytest.mark.gpu


def _routing(tokens, hidden, experts, topk, seed):
    dev = torch.device("cuda:0")
    g = torch.Generator(device=dev).manual_seed(seed)
    x = torch.randn(tokens, hidden, device=dev, dtype=torch.bfloat16, generator=g)
    w, idx = torch.topk(torch.softmax(torch.randn(tokens, experts, device=dev, generator=g), -1), topk, -1)
    return x, idx.contiguous(), w.float().contiguous()


@pytest.mark.parametrize("tokens", [1, 37, 700])
def test_gemm_on_another_stream_takes_this_steps_counts_and_rows(tokens):
    """``overlapped=True``: the GEMM derives the rows of an expert from the flags and counts of the dispatch."""
    H, E, K, N = 1024, 8, 4, 256
    dev = torch.device("cuda:0")
    b = Buffer(0, 1, E, H, tokens, K, device=dev, low_latency_mode=True, timeout_ms=1000)
    b.connect_ranks()
    wq, sw = quantize_weights(torch.randn(E, N, H, device=dev, generator=torch.Generator(device=dev).manual_seed(1)) * 0.05)
    side = torch.cuda.Stream(dev)
    for step in range(6):  # other counts in every step; each half of the double buffer three times
        x, idx, _ = _routing(max(1, tokens - 5 * step), H, E, K, step)
        side.wait_stream(torch.cuda.current_stream(dev))
        with torch.cuda.stream(side):
            (rx, sc), count, h, _, _ = b.low_latency_dispatch(x, idx)
        side.synchronize()
        flags = b._region(h.parity, "off_disp_flag", E * 8).view(torch.int64)
        assert bool((flags == h.epoch).all()) and int(b._region(h.parity, "off_counts_flag", 8).view(torch.int64)) == h.epoch
        want_count = torch.bincount(idx.reshape(-1), minlength=E).int()
        assert torch.equal(b._region(h.parity, "off_counts", E * 4).view(torch.int32), want_count) and torch.equal(count, want_count)
        a, sa = rx.view(-1, H), sc.view(-1, H // 128)
        status = torch.zeros(1, dtype=torch.int32, device=dev)
        got = grouped_gemm_fp8(a, sa, wq, sw, h.expert_offsets, count, status=status, fused_with=(b, h), overlapped=True, rows_per_expert=tokens)
        want = grouped_gemm_fp8(a, sa, wq, sw, h.expert_offsets, count, tile_mode=1)
        torch.cuda.synchronize()
        assert int(status) == 0 and b.status == 0
        for e, c in enumerate(want_count.tolist()):
            assert torch.equal(got[e * tokens : e * tokens + c], want[e * tokens : e * tokens + c]), (step, e, c)
    b.destroy()


def _one_phase(b, handle, phases, use_fp8=False):
    """The launch that the receive hook makes, on the current stream."""
    import ctypes

    from nixl_b200.ops import _lib

    p = b._disp_cache[(handle.parity, use_fp8, handle.rows_per_expert, False)][0]
    p.phases = phases
    _lib.check(b._dispatch_fn(ctypes.byref(p), _lib.raw_stream(b.device)), "dispatch")


def test_receive_phase_waits_for_the_flags():
    """A receive that runs before its rows are there must end in its bounded wait and say so, not hand out what is there."""
    T, H, E, K = 20, 512, 4, 2
    b = Buffer(0, 1, E, H, T, K, device=torch.device("cuda:0"), low_latency_mode=True, timeout_ms=50)
    b.connect_ranks()
    x, idx, _ = _routing(T, H, E, K, 2)
    recv, count, h, _, hook = b.low_latency_dispatch(x, idx, use_fp8=False, return_recv_hook=True)
    hook()
    torch.cuda.synchronize()
    assert b.status == 0 and torch.equal(count, torch.bincount(idx.reshape(-1), minlength=E).int())
    flags = b._region(h.parity, "off_disp_flag", E * 8).view(torch.int64)
    flags[1] = 0  # one expert's rows "not yet there"
    _one_phase(b, h, 2)
    torch.cuda.synchronize()
    assert b.status & 1 and int(b.mask[0]) == 1
    b.clean_mask_buffer()
    flags[1] = h.epoch
    _one_phase(b, h, 2)
    torch.cuda.synchronize()
    assert b.status == 0
    b.destroy()
