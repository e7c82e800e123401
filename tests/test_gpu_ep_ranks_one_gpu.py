"""Dispatch of a group of several ranks, one rank after the other on one GPU.

No kernel waits for another here: before a rank's dispatch runs, its buffer already holds what the peers would send it first,
their counts and flags, written by the host from the routing.  Each launch therefore passes its waits at once, sends its rows
to all buffers and ends.  When the last one has run every buffer must hold what a plain statement of the routing says, and
every arrival flag must be up."""
import ctypes

import pytest
import torch

from nixl_b200 import nixl_agent, nixl_agent_config
from nixl_b200.parallel import Buffer, per_token_cast_to_fp8

pytestmark = pytest.mark.gpu


def _ranks(n, experts, hidden, tokens, topk, tag, low_latency):
    dev = torch.device("cuda:0")
    bufs = []
    for r in range(n):
        agent = nixl_agent(f"{tag}_{r}", nixl_agent_config(enable_prog_thread=False, backends=["NVLINK"]))
        bufs.append(Buffer(r, n, experts, hidden, tokens, topk, device=dev, agent=agent, timeout_ms=1000, low_latency_mode=low_latency))
    md = [b.local_metadata() for b in bufs]
    for b in bufs:
        b.connect_ranks(metadata=md)
    return bufs


@pytest.mark.parametrize("num_sms", [0, 3])  # 3: several batches of tokens per CTA
@pytest.mark.parametrize("low_latency,kind", [(True, "fp8"), (False, "bf16"), (False, "ue8m0")])
@pytest.mark.parametrize("n,tokens,topk,hidden", [(4, 150, 6, 512), (3, 33, 1, 1536), (2, 700, 8, 2560)])
def test_dispatch_of_several_ranks(n, tokens, topk, hidden, low_latency, kind, num_sms):
    experts = 5 * n if topk < 6 else 8 * n
    bufs = _ranks(n, experts, hidden, tokens, topk, f"er{n}_{tokens}_{int(low_latency)}_{kind}_{num_sms}", low_latency)
    dev, El = torch.device("cuda:0"), experts // n
    xs, idxs, ws = [], [], []
    for r, b in enumerate(bufs):
        b.set_num_sms(num_sms)
        g = torch.Generator(device=dev).manual_seed(100 + r)
        t = tokens - 7 * r  # ranks differ in their number of tokens
        xs.append(torch.randn(t, hidden, device=dev, dtype=torch.bfloat16, generator=g))
        w, idx = torch.topk(torch.softmax(torch.randn(t, experts, device=dev, generator=g), -1), topk, -1)
        idx[::5, -1] = -1  # unused slots
        idxs.append(idx.contiguous())
        ws.append(w.float().contiguous())
    for step in (1, 2):  # both halves of the double buffer, and counters left clean by the first
        parity = step & 1
        counts = torch.stack([torch.bincount(i[i >= 0], minlength=experts) for i in idxs]).int()
        for b in bufs:
            b._region(parity, "off_counts", n * experts * 4).view(torch.int32).copy_(counts.reshape(-1))
            b._region(parity, "off_counts_flag", n * 8).view(torch.int64).fill_(step)
        results = []
        for r, b in enumerate(bufs):
            weights = ws[r] if not low_latency else None
            rpe = n * tokens if low_latency else 0
            results.append(b._dispatch(xs[r], idxs[r], kind != "bf16", False, rpe, 5, False, use_ue8m0=kind == "ue8m0", topk_weights=weights))  # send + publish, no wait for rows
        torch.cuda.synchronize()
        for d, b in enumerate(bufs):
            assert b.status == 0
            recv_x, scales, h, _, _ = results[d]
            flags = b._region(parity, "off_disp_flag", El * n * 8).view(torch.int64)
            assert bool((flags == step).all())
            offs, recv = h.expert_offsets.tolist(), h.recv_count.tolist()
            info = h.src_info.cpu()
            for le in range(El):
                e = d * El + le
                assert recv[le] == int(counts[:, e].sum())
                assert offs[le] == (le * n * tokens if low_latency else sum(recv[:le]))
                at = offs[le]
                for r in range(n):
                    c = int(counts[r, e])
                    assert int(h.layout_range[le, r]) == ((at - offs[le]) << 32) | c
                    rows = info[at : at + c]
                    assert bool((rows[:, 0] == r).all())
                    want = torch.nonzero(idxs[r].reshape(-1) == e).flatten().cpu()
                    assert torch.equal(torch.sort(rows[:, 1].long()).values, want)
                    t = (rows[:, 1].long() // topk).to(dev)
                    assert torch.equal(results[r][2].send_row.reshape(-1)[rows[:, 1].long().to(dev)].cpu(), torch.arange(at, at + c, dtype=torch.int32))
                    if kind == "bf16":
                        assert torch.equal(recv_x[at : at + c], xs[r][t])
                    elif c:
                        q, s = per_token_cast_to_fp8(xs[r], round_scale=kind == "ue8m0")
                        if kind == "ue8m0":
                            assert torch.equal(scales[at : at + c].view(torch.uint8).int(), ((s[t].view(torch.int32) >> 23) & 255))
                            assert torch.equal(recv_x[at : at + c].view(torch.uint8), q[t].view(torch.uint8))
                        else:  # x * (448 / amax): PyTorch multiplies by a reciprocal, so a code may differ by a step on a boundary
                            torch.testing.assert_close(scales[at : at + c], s[t], rtol=1e-6, atol=0)
                            diff = (recv_x[at : at + c].view(torch.uint8).int() - q[t].view(torch.uint8).int()).abs()
                            assert int(diff.max()) <= 1 and float((diff > 0).float().mean()) < 0.02
                    at += c
            if not low_latency:  # group records of the rank-reduced combine
                rec = b._region(parity, "off_grp", n * tokens * 80).view(torch.int32).view(n, tokens, 20).cpu()
                for r in range(n):
                    send = results[r][2].send_row.cpu()
                    here = (idxs[r] // El == d).cpu() & (idxs[r] >= 0).cpu()
                    for t in range(idxs[r].shape[0]):
                        ks = torch.nonzero(here[t]).flatten()
                        if len(ks) == 0:
                            continue
                        m = len(ks)
                        assert rec[r, t, 0] == m and rec[r, t, 1] == step
                        assert torch.equal(rec[r, t, 4 : 4 + m], send[t, ks])
                        assert torch.equal(rec[r, t, 12 : 12 + m].view(torch.float32), ws[r].cpu()[t, ks])
    for b in bufs:
        b.destroy()


# 12 bytes per expert: below and just above 48 KiB, more than 16 bytes per expert would leave room for, and (8 bytes) more than 12 would
@pytest.mark.parametrize("n", [6, 9, 30, 40])
def test_dispatch_with_more_experts_than_the_default_shared_memory_holds(n):
    El, tokens, topk, hidden = 512, 40, 4, 512
    experts = n * El
    bufs = _ranks(n, experts, hidden, tokens, topk, f"er_many{n}", False)
    dev = torch.device("cuda:0")
    g = torch.Generator(device=dev).manual_seed(5)
    xs = [torch.randn(tokens, hidden, device=dev, dtype=torch.bfloat16, generator=g) for _ in bufs]
    idxs = [torch.topk(torch.randn(tokens, experts, device=dev, generator=g), topk, -1)[1].contiguous() for _ in bufs]
    counts = torch.stack([torch.bincount(i.reshape(-1), minlength=experts) for i in idxs]).int()
    for b in bufs:
        b._region(1, "off_counts", n * experts * 4).view(torch.int32).copy_(counts.reshape(-1))
        b._region(1, "off_counts_flag", n * 8).view(torch.int64).fill_(1)
    results = [b._dispatch(xs[r], idxs[r], False, False, 0, 5, False) for r, b in enumerate(bufs)]
    torch.cuda.synchronize()
    for d, b in enumerate(bufs):
        assert b.status == 0
        recv_x, _, h, _, _ = results[d]
        mine = counts[:, d * El : (d + 1) * El].sum(0).int()
        assert torch.equal(h.recv_count, mine)
        for r in range(n):
            t, k = torch.nonzero(idxs[r] // El == d, as_tuple=True)
            rows = results[r][2].send_row[t, k].long()
            assert torch.equal(recv_x[rows], xs[r][t])
            assert bool((rows >= h.expert_offsets[idxs[r][t, k] - d * El]).all())
    for b in bufs:
        b.destroy()


@pytest.mark.parametrize("mode", ["push", "pull", "reduced"])
@pytest.mark.parametrize("tokens,topk,experts,hidden", [(1, 1, 1, 512), (7, 3, 4, 512), (130, 8, 16, 2048), (1300, 4, 8, 1024), (40, 12, 16, 512)])
def test_combine_of_one_rank(tokens, topk, experts, hidden, mode):
    """One rank that holds every expert sums its rows in place; every mode must give the fp32 sum, rounded once."""
    if mode == "reduced" and topk > 8:
        pytest.skip("group records hold eight copies")
    dev = torch.device("cuda:0")
    low_latency = mode != "reduced"
    b = Buffer(0, 1, experts, hidden, tokens, topk, device=dev, low_latency_mode=low_latency)
    b.connect_ranks()
    g = torch.Generator(device=dev).manual_seed(tokens)
    x = torch.randn(tokens, hidden, device=dev, dtype=torch.bfloat16, generator=g)
    w, idx = torch.topk(torch.softmax(torch.randn(tokens, experts, device=dev, generator=g), -1), topk, -1)
    idx[::3, 0] = -1
    if tokens > 2:
        idx[2] = -1  # a token without experts
    idx, w = idx.contiguous(), w.float().contiguous()
    for _ in range(3):
        if low_latency:
            recv, _, h, _, _ = b.low_latency_dispatch(x, idx, use_fp8=False)
            flat = recv.view(-1, hidden)
        else:
            flat, _, h = b.dispatch(x, idx, use_fp8=False, topk_weights=w)
        y = torch.full_like(flat, float("nan"))  # rows that no copy fills are never read
        for e in range(experts):
            s, c = int(h.expert_offsets[e]), int(h.recv_count[e])
            y[s : s + c] = (flat[s : s + c].float() * (e + 1)).to(torch.bfloat16)
        if mode == "pull":
            buf = b.get_next_combine_buffer(h)
            buf.view(-1, hidden)[: y.shape[0]].copy_(y)
            out, _, hook = b.low_latency_combine(buf, idx, w, h, zero_copy=True, return_recv_hook=True)
            hook()
        elif mode == "push":
            out, _, hook = b.low_latency_combine(y.view(experts, -1, hidden), idx, w, h, return_recv_hook=True)
            y.fill_(float("nan"))  # the send phase is over: the caller may overwrite its rows
            hook()
        else:
            out = b.combine(y, idx, w, h)
        want = torch.zeros(tokens, hidden, device=dev, dtype=torch.float64)
        mass = torch.zeros_like(want)
        for k in range(topk):
            on = (idx[:, k] >= 0).double().unsqueeze(1)
            term = (x.float() * (idx[:, k] + 1).unsqueeze(1)).to(torch.bfloat16).double() * w[:, k].double().unsqueeze(1) * on
            want += term
            mass += term.abs()
        # one rounding to bf16 (half a step, 2^-9 of the value) of a sum of up to 12 fp32 products
        assert bool(((out.double() - want).abs() <= want.abs() * 2.0**-8 + mass * (16 * 2.0**-24)).all())
    assert b.status == 0
    b.destroy()


@pytest.mark.parametrize("low_latency", [True, False])
def test_fused_gemm_takes_the_scales_that_arrive(low_latency):
    """The GEMM that overlaps a dispatch must read a row's scales after the row's arrival flag, not what the buffer held
    before: the scale area is filled with another value first, in both halves."""
    from nixl_b200.ops import grouped_gemm_fp8, quantize_weights

    T, H, E, K, N = 200, 2048, 8, 4, 512
    dev = torch.device("cuda:0")
    g = torch.Generator(device=dev).manual_seed(3)
    b = Buffer(0, 1, E, H, T, K, device=dev, low_latency_mode=low_latency)
    b.connect_ranks()
    x = torch.randn(T, H, device=dev, generator=g).to(torch.bfloat16)
    _, idx = torch.topk(torch.softmax(torch.randn(T, E, device=dev, generator=g), -1), K, -1)
    idx = idx.contiguous()
    wq, sw = quantize_weights(torch.randn(E, N, H, device=dev, generator=g) * 0.05)
    rows = b.ll_rows if low_latency else b.compact_rows
    for _ in range(4):
        for parity in (0, 1):
            b._region(parity, "off_recv_scales", rows * (H // 128) * 4).view(torch.float32).fill_(1.0e4)
        torch.cuda.synchronize()
        got, h, rx, sc = b.dispatch_gemm(x, idx, wq, sw, low_latency=low_latency)
        torch.cuda.synchronize()
        want = grouped_gemm_fp8(rx[:rows], sc[:rows], wq, sw, h.expert_offsets, h.recv_count, tile_mode=1)
        torch.cuda.synchronize()
        for e in range(E):
            s, c = int(h.expert_offsets[e]), int(h.recv_count[e])
            assert torch.equal(got[s : s + c], want[s : s + c]), (e, c)
    b.destroy()
