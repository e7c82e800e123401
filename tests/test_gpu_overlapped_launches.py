"""Kernels whose launch overlaps the end of the kernel in front of them: results, and the room that they leave to others.

No kernel here waits for another that runs beside it: a wait that is meant to last ends at its own limit."""
import ctypes
import time

import pytest
import torch

from nixl_b200 import nixl_agent, nixl_agent_config
from nixl_b200.ops import KVLayout, KVTransfer, _lib, grouped_gemm_fp8, grouped_gemm_mxfp8, quantize_weights, quantize_weights_ue8m0
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


# Few rows per expert (W on the MMA's M side), more, CTA pairs, block-scaled.
@pytest.mark.parametrize("tokens,low_latency,kind", [(24, True, "fp8"), (128, True, "fp8"), (700, False, "fp8"), (24, False, "mx"), (700, False, "mx")])
def test_dispatch_gemm_combine_without_a_pause(tokens, low_latency, kind):
    """Inputs, routing and the experts' weights are other ones in every step, each written by the kernel in front of the one that
    reads it.  The results are those of the same calls with the GPU at rest between them."""
    H, E, K, steps = 1024, 8, 4, 8
    dev = torch.device("cuda:0")
    b = Buffer(0, 1, E, H, tokens, K, device=dev, low_latency_mode=low_latency, timeout_ms=1000)
    b.connect_ranks()
    given = [_routing(tokens, H, E, K, 200 + i) for i in range(steps)]
    g = torch.Generator(device=dev).manual_seed(5)
    quantize = quantize_weights if kind == "fp8" else quantize_weights_ue8m0
    weights = [quantize(torch.randn(E, H, H, device=dev, generator=g) * 0.05 * 2.0**i) for i in range(steps)]
    x, idx, w = (torch.empty_like(t) for t in given[0])
    wq, sw = (torch.empty_like(t) for t in weights[0])
    rows = b.ll_rows if low_latency else b.compact_rows
    y = torch.zeros(rows, H, device=dev, dtype=torch.bfloat16)
    status = torch.zeros(1, dtype=torch.int32, device=dev)
    results = []
    for pause in (True, False):
        outs = []

        def done():
            if pause:
                torch.cuda.synchronize()

        torch.cuda.synchronize()
        for i in range(steps):
            w.copy_(given[i][2])
            idx.copy_(given[i][1])
            x.copy_(given[i][0])
            done()
            if low_latency:
                (rx, sc), _, h, _, _ = b.low_latency_dispatch(x, idx)
            else:
                rx, sc, h = b.dispatch(x, idx, use_ue8m0=kind == "mx", topk_weights=w)
            done()
            wq.view(torch.uint8).copy_(weights[i][0].view(torch.uint8))
            sw.copy_(weights[i][1])
            done()
            if kind == "mx":
                grouped_gemm_mxfp8(rx, sc, wq, sw, h.expert_offsets, h.recv_count, out=y, status=status)
            else:
                grouped_gemm_fp8(rx.view(-1, H), sc.view(-1, H // 128), wq, sw, h.expert_offsets, h.recv_count, out=y, status=status)
            done()
            outs.append(b.combine(y, idx, w, h) if not low_latency else b.low_latency_combine(y, idx, w, h)[0])
            done()
        torch.cuda.synchronize()
        assert b.status == 0 and int(status) == 0
        results.append(outs)
    for i, (apart, chained) in enumerate(zip(*results)):
        assert bool(apart.isfinite().all()) and torch.equal(apart, chained), i
    b.destroy()


@pytest.mark.parametrize("fp8", [False, True])
def test_kv_transfers_that_read_what_the_one_in_front_wrote(fp8):
    """Two hand-overs, the second from the first one's destination, with block tables that are written right in front of each."""
    dev = torch.device("cuda:0")
    cfg = nixl_agent_config(enable_prog_thread=False, backends=["NVLINK"])
    a, b, c = (nixl_agent(f"kvchain{int(fp8)}_{r}", cfg) for r in "abc")
    blocks, heads, tensors, pairs, steps = 96, 4, 6, 70, 10
    g = torch.Generator(device=dev).manual_seed(4)

    def caches(dtype):
        return [torch.zeros(blocks, 16, heads, 128, device=dev, dtype=dtype) for _ in range(tensors)]

    src, mid, dst = caches(torch.bfloat16), caches(torch.bfloat16), caches(torch.uint8 if fp8 else torch.bfloat16)
    for t in src:
        t.copy_(torch.randn(t.shape, device=dev, generator=g))
    for agent, mem in ((a, src), (b, mid), (c, dst)):
        agent.register_memory(mem)
    a.add_remote_agent(b.get_agent_metadata())
    b.add_remote_agent(c.get_agent_metadata())

    def remote(ts):
        return [(t.data_ptr(), t.numel() * t.element_size(), t.get_device()) for t in ts]

    layout = KVLayout(16, heads, 128)
    first = KVTransfer(a, src, layout, b.name, remote(mid), layout)
    second = KVTransfer(b, mid, layout, c.name, remote(dst), KVLayout(16, heads, 128, elem_bytes=1 if fp8 else 2), cast_fp8=fp8)
    ids = [[torch.randperm(blocks, device=dev, generator=g)[:pairs].int() for _ in range(3)] for _ in range(steps)]
    tables = [torch.zeros(pairs, dtype=torch.int32, device=dev) for _ in range(4)]
    torch.cuda.synchronize()
    for one, two, three in ids:
        tables[1].copy_(two)
        tables[0].copy_(one)
        first.post(tables[0], tables[1])
        tables[3].copy_(three)
        tables[2].copy_(two)
        last = second.post(tables[2], tables[3])
    second.wait(last)
    torch.cuda.synchronize()
    for s, m, d in zip(src, mid, dst):
        want_m, want_d = torch.zeros_like(m), torch.zeros_like(d)
        for one, two, three in ids:
            want_m[two.long()] = s[one.long()]
            moved = want_m[two.long()]
            want_d[three.long()] = moved.to(torch.float8_e4m3fn).view(torch.uint8) if fp8 else moved
        assert torch.equal(m, want_m) and torch.equal(d, want_d)
    first.close()
    second.close()


@pytest.mark.parametrize("rows_each", [8, 64, 300])
def test_gemms_in_a_graph(rows_each):
    """Captured launches overlap as eager ones do; the second GEMM's weights are written in front of it."""
    dev = torch.device("cuda:0")
    G, N, K = 8, 1024, 1024
    g = torch.Generator(device=dev).manual_seed(6)
    a, sa = per_token_cast_to_fp8(torch.randn(G * rows_each, K, device=dev, generator=g).to(torch.bfloat16))
    weights = [quantize_weights(torch.randn(G, N, K, device=dev, generator=g) * 0.05 * (i + 1)) for i in range(3)]
    wq, sw = (torch.empty_like(t) for t in weights[0])
    other, other_scale = (torch.empty_like(t) for t in weights[0])
    rs = torch.arange(G, device=dev, dtype=torch.int32) * rows_each
    rc = torch.full_like(rs, rows_each)
    outs = [torch.empty(G * rows_each, N, device=dev, dtype=torch.bfloat16) for _ in range(2)]
    status = torch.zeros(1, dtype=torch.int32, device=dev)

    def both():
        grouped_gemm_fp8(a, sa, wq, sw, rs, rc, out=outs[0], status=status)
        wq.view(torch.uint8).copy_(other.view(torch.uint8))
        sw.copy_(other_scale)
        grouped_gemm_fp8(a, sa, wq, sw, rs, rc, out=outs[1], status=status)

    def fill(i):
        for to, of in zip((wq, other), (weights[i][0], weights[(i + 1) % 3][0])):
            to.view(torch.uint8).copy_(of.view(torch.uint8))
        sw.copy_(weights[i][1])
        other_scale.copy_(weights[(i + 1) % 3][1])

    want = []
    for i in range(3):
        fill(i)
        both()
        want.append([t.clone() for t in outs])
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        both()
    for i in (2, 0, 1):
        fill(i)
        graph.replay()
        torch.cuda.synchronize()
        assert int(status) == 0 and all(torch.equal(got, ref) for got, ref in zip(outs, want[i]))
    assert not torch.equal(want[0][0], want[0][1])


def test_an_sm_that_a_gemm_has_left_is_split_anew():
    """A GEMM's ring leaves an SM next to no L1.  A kernel that moves in behind it needs L1 for its loads in flight: overlapping the
    GEMM's end must not cost it more than a launch of its own.  (It cost 6 us more where the SMs stayed as the GEMM had them, and
    takes 2 us less where they do not; the line lies at half of that cost.)"""
    T, H, E, K, depth = 4096, 4096, 32, 8, 512
    dev = torch.device("cuda:0")
    b = Buffer(0, 1, E, H, T, K, device=dev, low_latency_mode=False, timeout_ms=1000)
    b.connect_ranks()
    x, idx, w = _routing(T, H, E, K, 1)
    recv, scales, h = b.dispatch(x, idx, use_ue8m0=True, topk_weights=w)
    a, sa = recv[:, :depth].contiguous(), scales.view(torch.int32)[:, : depth // 512].contiguous()
    wq, sw = quantize_weights_ue8m0(torch.randn(E, H, depth, device=dev) * 0.05)
    y, out, pad = b.get_next_combine_buffer(h).view(-1, H), torch.empty_like(x), torch.zeros(1, device=dev)
    status = torch.zeros(1, dtype=torch.int32, device=dev)

    def step(apart):
        grouped_gemm_mxfp8(a, sa, wq, sw, h.expert_offsets, h.recv_count, out=y, status=status)
        if apart:
            pad.zero_()  # a kernel that neither lets another in nor moves in early
        b.combine(y, idx, w, h, out=out)

    times = {False: [], True: []}
    for i in range(42):
        for apart in times:
            begin, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            torch.cuda._sleep(200000)  # all launches are queued when the first one starts
            begin.record()
            step(apart)
            end.record()
            end.synchronize()
            if i > 1:
                times[apart].append(begin.elapsed_time(end) * 1e3)
    chained, separate = (sorted(times[apart])[20] for apart in (False, True))
    assert b.status == 0 and int(status) == 0
    assert chained < separate + 3, (chained, separate)
    b.destroy()
