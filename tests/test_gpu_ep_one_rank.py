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
        assert count._nixl_expected_rows == idx.numel()  # by which a GEMM chooses its tiles
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


def _dispatched(b, x, idx, w, low_latency):
    """Rows as the experts left them (scaled by expert number + 1) and the sum they must give, with the bound of its rounding."""
    if low_latency:
        recv, _, h, _, _ = b.low_latency_dispatch(x, idx, use_fp8=False)
    else:
        recv, _, h = b.dispatch(x, idx, use_fp8=False, topk_weights=w)
    flat = recv.view(-1, x.shape[1])
    y = flat.clone()
    for e in range(b.num_experts):
        s, c = int(h.expert_offsets[e]), int(h.recv_count[e])
        y[s : s + c] = (flat[s : s + c].float() * (e + 1)).to(torch.bfloat16)
    want = torch.zeros(x.shape, device=x.device, dtype=torch.float64)
    mass = torch.zeros_like(want)
    for k in range(idx.shape[1]):
        term = (x.float() * (idx[:, k] + 1).unsqueeze(1)).to(torch.bfloat16).double() * w[:, k].double().unsqueeze(1) * (idx[:, k] >= 0).unsqueeze(1)
        want += term
        mass += term.abs()
    # one rounding to bf16 (half a step, 2^-9 of the value) of a sum of up to 8 fp32 products
    return y, h, want, want.abs() * 2.0**-8 + mass * (16 * 2.0**-24)


@pytest.mark.parametrize("mode", ["push", "pull", "reduced", "coded"])
@pytest.mark.parametrize("at", [None, 0, 3, -2])  # out: elsewhere; at a row of x; two rows in front of x
@pytest.mark.parametrize("tokens", [1, 130, 900])
def test_combine_into_the_rows_it_reads(mode, at, tokens):
    """Only x's own rows may be read before all of x has been: `out` may overlap x where nothing is loaded from x in place."""
    H, E, K = 1024, 8, 4
    dev = torch.device("cuda:0")
    low_latency = mode != "reduced"
    b = Buffer(0, 1, E, H, tokens, K, device=dev, low_latency_mode=low_latency)
    b.connect_ranks()
    for step in range(3):
        x, idx, w = _routing(tokens, H, E, K, step)
        idx[::3, 0] = -1
        y, h, want, bound = _dispatched(b, x, idx, w, low_latency)
        room = torch.empty(y.shape[0] + tokens + 8, H, device=dev, dtype=torch.bfloat16)
        rows = room[2 : 2 + y.shape[0]]
        rows.copy_(y)
        out = None if at is None else room[2 + at : 2 + at + tokens]
        if mode == "coded":
            apart, _, _ = b.low_latency_combine(y, idx, w, h, use_logfmt=True)
            got, _, _ = b.low_latency_combine(rows, idx, w, h, use_logfmt=True, out=out)
            assert torch.equal(got, apart)
            continue
        if mode == "reduced":
            got = b.combine(rows, idx, w, h, out=out)
        else:  # pull: from rows outside the exposed region, which are staged there first
            b.combine_pull = mode == "pull"
            got, _, _ = b.low_latency_combine(rows, idx, w, h, out=out)
        assert out is None or got.data_ptr() == out.data_ptr()
        assert bool(((got.double() - want).abs() <= bound).all())
    assert b.status == 0
    b.destroy()


@pytest.mark.parametrize("mode", ["push", "pull", "coded"])
def test_combine_with_a_hook_writes_out_in_the_hook(mode):
    T, H, E, K = 50, 1024, 8, 4
    b = Buffer(0, 1, E, H, T, K, device=torch.device("cuda:0"), low_latency_mode=True)
    b.connect_ranks()
    x, idx, w = _routing(T, H, E, K, 5)
    y, h, want, bound = _dispatched(b, x, idx, w, True)
    coded = mode == "coded"
    if mode == "pull":
        b.get_next_combine_buffer(h).view(-1, H).copy_(y)
        y = b.get_next_combine_buffer(h).view(-1, H)
    now, _, _ = b.low_latency_combine(y, idx, w, h, use_logfmt=coded, zero_copy=mode == "pull")
    out = torch.full((T, H), 7.0, device=x.device, dtype=torch.bfloat16)
    got, _, hook = b.low_latency_combine(y, idx, w, h, use_logfmt=coded, zero_copy=mode == "pull", return_recv_hook=True, out=out)
    torch.cuda.synchronize()
    assert bool((out == 7.0).all())
    if mode != "pull":
        y.fill_(float("nan"))  # the send phase has read them
    hook()
    torch.cuda.synchronize()
    assert torch.equal(out, now) and b.status == 0
    if not coded:
        assert bool(((out.double() - want).abs() <= bound).all())
    b.destroy()


def test_rank_reduced_combine_leaves_out_tokens_without_experts():
    """Tokens whose slots the caller took out after the dispatch come back as zeros."""
    T, H, E, K = 70, 1024, 8, 3
    b = Buffer(0, 1, E, H, T, K, device=torch.device("cuda:0"))
    b.connect_ranks()
    x, idx, w = _routing(T, H, E, K, 9)
    y, h, want, bound = _dispatched(b, x, idx, w, False)
    fewer = idx.clone()
    fewer[::4] = -1
    fewer[1::4, 0] = -1  # (one slot: the recorded sum of the token stays)
    got = b.combine(y, fewer, w, h)
    assert bool((got[::4] == 0).all())
    want[::4] = 0
    assert bool(((got.double() - want).abs() <= bound).all())
    overlapping = b.combine(y, fewer, w, h, out=y[1 : 1 + T])  # the path of larger groups
    assert torch.equal(overlapping, got)
    b.destroy()


@pytest.mark.parametrize("tokens,experts,topk,sms", [(1, 5, 1, 0), (70, 33, 4, 1), (150, 100, 8, 2), (700, 64, 3, 0), (2500, 32, 8, 0)])
def test_compact_dispatch_places_every_copy_once(tokens, experts, topk, sms):
    """Few CTAs (several batches of tokens each), more experts than a warp's width, slots without an expert."""
    H = 512
    b = Buffer(0, 1, experts, H, tokens, topk, device=torch.device("cuda:0"), low_latency_mode=False, timeout_ms=1000)
    b.connect_ranks()
    b.set_num_sms(sms)
    for step in range(3):
        x, idx, w = _routing(tokens, H, experts, topk, 10 + step)
        idx[step::7] = -1
        recv, _, h = b.dispatch(x, idx, use_fp8=False, topk_weights=w)
        torch.cuda.synchronize()
        assert b.status == 0
        want = torch.bincount(idx[idx >= 0], minlength=experts)
        start = torch.cumsum(want, 0) - want
        assert torch.equal(h.recv_count, want.int()) and torch.equal(h.expert_offsets[:experts], start.int())
        assert int(h.expert_offsets[experts]) == int(want.sum())
        flags = b._region(h.parity, "off_disp_flag", experts * 8).view(torch.int64)
        assert bool((flags == h.epoch).all()) and int(b._region(h.parity, "off_counts_flag", 8).view(torch.int64)) == h.epoch
        t, k = torch.nonzero(idx >= 0, as_tuple=True)
        rows = h.send_row[t, k].long()
        assert torch.equal(torch.sort(rows).values, torch.arange(rows.numel(), device=rows.device))  # each row once
        assert bool(((rows >= start[idx[t, k]]) & (rows < (start + want)[idx[t, k]])).all())          # among its expert's
        assert torch.equal(recv[rows], x[t])
        assert torch.equal(h.src_info[rows, 1].long(), t * topk + k)
    b.destroy()


def _compact(b, x, idx, w):
    """A compact dispatch, every copy of which must have arrived in a row of its own among its expert's."""
    recv, _, h = b.dispatch(x, idx, use_fp8=False, topk_weights=w)
    t, k = torch.nonzero(idx >= 0, as_tuple=True)

    def check():
        want = torch.bincount(idx[idx >= 0], minlength=b.num_experts)
        rows = h.send_row[t, k].long()
        return (torch.equal(h.recv_count, want.int()) and torch.equal(torch.sort(rows).values, torch.arange(rows.numel(), device=rows.device))
                and torch.equal(recv[rows], x[t]))

    return recv, h, check


def test_dispatch_leaves_the_barrier_of_a_combine_alone():
    """A combine on another stream may have CTAs at its grid barrier while a dispatch begins and ends: the dispatch must neither
    count them as its own nor send them away."""
    H, E, K, T = 512, 32, 4, 700
    b = Buffer(0, 1, E, H, T, K, device=torch.device("cuda:0"), low_latency_mode=False, timeout_ms=1000)
    b.connect_ranks()
    arrivals, generation = 1000, 9  # more than a dispatch has CTAs
    b._bar[0], b._bar[1] = arrivals, generation
    for step in range(4):
        x, idx, w = _routing(T - 50 * step, H, E, K, 30 + step)
        _, _, check = _compact(b, x, idx, w)
        torch.cuda.synchronize()
        assert b.status == 0 and check()
        assert b._bar.tolist() == [arrivals, generation, 0, 0]
    b.destroy()


@pytest.mark.parametrize("mode", ["push", "reduced"])
def test_dispatch_beside_a_combine_of_the_same_buffer(mode):
    """Step n + 1 is dispatched on one stream while step n is combined on another, into memory that overlaps its input (the path of
    larger groups, with a grid barrier).  Neither waits for the other, and there is room for both at once."""
    H, E, K, T = 1024, 32, 8, 900
    dev = torch.device("cuda:0")
    b = Buffer(0, 1, E, H, T, K, device=dev, low_latency_mode=False, timeout_ms=1000)
    b.connect_ranks()
    b.set_num_sms(32)
    sends, returns = torch.cuda.Stream(dev), torch.cuda.Stream(dev)
    inputs = [_routing(T - 11 * i, H, E, K, 60 + i) for i in range(4)]
    alone = []
    for x, idx, w in inputs:
        recv, _, h = b.dispatch(x, idx, use_fp8=False, topk_weights=w if mode == "reduced" else None)
        alone.append(b.combine(recv.clone(), idx, w, h).clone())
    rooms = [torch.empty(b.compact_rows + T, H, device=dev, dtype=torch.bfloat16) for _ in range(2)]
    torch.cuda.synchronize()
    combined = None
    results, dispatched, keep = [], [], []
    for step in range(16):
        x, idx, w = inputs[step % 4]
        with torch.cuda.stream(sends):
            if combined is not None and step >= 2:
                sends.wait_event(combined[step - 2])  # the half of the double buffer that this step takes is free again
            recv, _, h = b.dispatch(x, idx, use_fp8=False, topk_weights=w if mode == "reduced" else None)
            dispatched.append((recv, h, sends.record_event()))
        with torch.cuda.stream(returns):
            returns.wait_event(dispatched[step][2])
            y = rooms[step % 2][T:]
            y.copy_(recv)
            got = b.combine(y, idx, w, h, out=rooms[step % 2][T - 5 : 2 * T - 5][: x.shape[0]])
            results.append(got.clone())
            combined = (combined or []) + [returns.record_event()]
            keep.append(b._keep_c)
    torch.cuda.synchronize()
    assert b.status == 0 and b._bar.tolist()[0] == 0 and b._bar.tolist()[2:] == [0, 0]
    for step, got in enumerate(results):
        err = (got.double() - alone[step % 4].double()).norm() / alone[step % 4].double().norm()
        assert float(err) < 2.0**-8, (step, float(err))  # (rows may come in another order, and with it the sum's; half a bf16 step)
    b.destroy()


@pytest.mark.parametrize("low_latency", [True, False])
def test_rows_are_announced_while_the_dispatch_for_a_fused_gemm_runs(low_latency):
    """``dispatch_gemm``'s GEMM takes an expert's rows as they arrive: counts and flags go up long before the last row is sent."""
    T, H, E, K = 4096, 4096, 16, 8
    dev = torch.device("cuda:0")
    b = Buffer(0, 1, E, H, T, K, device=dev, low_latency_mode=low_latency, timeout_ms=1000)
    b.connect_ranks()
    x, _, _ = _routing(T, H, E, K, 1)
    idx = torch.arange(K, 2 * K, device=dev).repeat(T, 1)
    idx[:64] -= K  # experts 0 to 7 get the first tokens, 8 to 15 the others
    looks, seen = torch.cuda.Stream(dev), torch.empty(E + 1, dtype=torch.int64).pin_memory()
    for step in range(3):
        parity = (b.epoch + 1) & 1
        flags, counts_flag = b._region(parity, "off_disp_flag", E * 8).view(torch.int64), b._region(parity, "off_counts_flag", 8).view(torch.int64)
        torch.cuda.synchronize()
        _, _, h, _, _ = b._dispatch(x, idx, True, False, T if low_latency else 0, 5, False, grid=1)  # as dispatch_gemm launches it; one CTA: milliseconds
        done = torch.cuda.Event()
        done.record()
        early = torch.zeros(E + 1, dtype=torch.bool)
        while True:
            with torch.cuda.stream(looks):
                seen[:E].copy_(flags, non_blocking=True)
                seen[E:].copy_(counts_flag, non_blocking=True)
            looks.synchronize()
            if done.query():
                break
            early |= seen == h.epoch
        assert step == 0 or (bool(early[:K].all()) and bool(early[E])), early.tolist()  # (the first launch loads the kernel)
        assert b.status == 0 and bool((flags == h.epoch).all()) and b._cnt.count_nonzero() == 0
        assert torch.equal(h.recv_count, torch.bincount(idx.reshape(-1), minlength=E).int())
    b.destroy()
