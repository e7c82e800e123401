"""The work that programs have this framework do on one GPU, as cases that can be timed and compared.

Four families, each through its public entry points:

* ``xfer``    descriptor transfers between two agents (``nixl_agent.transfer`` / ``check_xfer_state``);
* ``blocks``  a request for numbered cache blocks, built and posted per request (``KVBlockTransfer``);
* ``kv``      the fused paged-KV transfer (``KVTransfer``): gather, head regrouping, optional fp8 cast, scatter;
* ``ep``, ``moe``, ``gemm``  the expert-parallel path: dispatch and combine with experts that return their input,
  dispatch -> expert GEMM -> combine, and the grouped GEMM by itself.

On one GPU both ends of a transfer lie in the same memory and an expert-parallel group has one rank that holds all
experts of the case (as many as a rank of a larger group would hold).
"""
import math

import numpy as np
import torch

from nixl_b200 import nixl_agent, nixl_agent_config
from nixl_b200.ops import (KVBlockTransfer, KVLayout, KVTransfer, describe_blocks, grouped_gemm_fp8, grouped_gemm_mxfp8, quantize_weights,
                           quantize_weights_ue8m0, to_ue8m0)
from nixl_b200.parallel import Buffer

KIB, MIB = 1 << 10, 1 << 20


def listed():
    return [
        # The smallest call: one 4 KiB block written to a peer and waited for (a control message, one small cache page).
        # What counts is the time from the post to the completion seen by the caller.
        {"name": "write_4k", "family": "xfer", "op": "WRITE", "descs": 1, "bytes": 4 * KIB, "align": 256, "ragged": False, "host": False},
        # An ordinary request: 256 cache blocks of 64 KiB, scattered at the receiver.
        {"name": "write_256x64k", "family": "xfer", "op": "WRITE", "descs": 256, "bytes": 64 * KIB, "align": 256, "ragged": False, "host": False},
        # Slices of 16-bit tensors of all lengths, fetched from a peer into a packed buffer: lengths and offsets are even and otherwise arbitrary.
        {"name": "read_ragged_512", "family": "xfer", "op": "READ", "descs": 512, "bytes": 64 * KIB, "align": 2, "ragged": True, "host": False},
        # The largest: the benchmark's request of 16 x 64 MiB, destination blocks in another order than the source's.
        {"name": "write_16x64m", "family": "xfer", "op": "WRITE", "descs": 16, "bytes": 64 * MIB, "align": 256, "ragged": False, "host": False},
        # A serving engine's request by block numbers, new ones each time: K and V of 32 layers, 32 blocks of 16 tokens x 8 heads x 128.
        {"name": "blocks_64x32", "family": "blocks", "tensors": 64, "blocks": 32, "pool": 256, "block_bytes": 32 * KIB, "op": "WRITE"},
        # Prefill at TP4 to decode at TP2: a prompt of 4096 tokens, 2 of 8 KV heads, 32 layers.
        {"name": "kv_bf16_4096", "family": "kv", "tensors": 64, "pairs": 256, "pool": 512, "tokens": 16, "heads": 2, "dst_heads": 4, "dim": 128,
         "src_order": "NHD", "dst_order": "NHD", "fp8": False},
        # A shorter, odd prompt with 64-wide heads: 61 blocks, 24 layers, cast to fp8 and turned from token-major to head-major on the way.
        {"name": "kv_fp8_hnd_976", "family": "kv", "tensors": 48, "pairs": 61, "pool": 128, "tokens": 16, "heads": 8, "dst_heads": 8, "dim": 64,
         "src_order": "NHD", "dst_order": "HND", "fp8": True},
        # A decode step's all-to-all without its experts: 128 tokens, top-8 of 32 local experts, low-latency layout, bf16.
        {"name": "ep_decode_128", "family": "ep", "tokens": 128, "hidden": 7168, "experts": 32, "topk": 8, "low_latency": True, "logfmt": False},
        # A prefill step's: 4096 tokens, compact layout, rank-reduced combine.
        {"name": "ep_prefill_4096", "family": "ep", "tokens": 4096, "hidden": 7168, "experts": 32, "topk": 8, "low_latency": False, "logfmt": False},
        # A whole decode step: fp8 dispatch, expert GEMM (about 32 rows per expert, so the weights are what is read), combine in place.
        {"name": "moe_decode_128", "family": "moe", "tokens": 128, "hidden": 4096, "experts": 32, "topk": 8, "low_latency": True},
        # A whole prefill step: fp8 dispatch with power-of-two scales, block-scaled expert GEMM, rank-reduced combine.
        {"name": "moe_prefill_4096", "family": "moe", "tokens": 4096, "hidden": 4096, "experts": 32, "topk": 8, "low_latency": False},
        # The expert up-projection of a prefill step by itself, fp32 block scales, rows per expert as routing leaves them.
        {"name": "gemm_fp8_16384", "family": "gemm", "groups": 32, "rows": 16384, "n": 2048, "k": 7168, "mx": False},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    family = rng.choice(["xfer", "xfer", "xfer", "blocks", "kv", "kv", "ep", "ep", "moe", "gemm", "gemm"])
    if family == "xfer":
        host = rng.random() < 0.15
        align = rng.choice([1, 2, 16, 256, 256])
        total = _log(rng, 1 * KIB, (8 if host else 48 if align < 16 else 1024) * MIB)
        descs = min(_log(rng, 1, 2048), max(1, total // 64))
        size = max(1, total // descs)
        if align > 2 and rng.random() < 0.7:
            size = max(align, size // align * align)
        return {"family": "xfer", "op": rng.choice(["WRITE", "READ"]), "descs": descs, "bytes": size, "align": align,
                "ragged": rng.random() < 0.4, "host": host}
    if family == "blocks":
        blocks = _log(rng, 1, 48)
        return {"family": "blocks", "tensors": rng.choice([1, 2, 24, 36, 48, 61, 64]), "blocks": blocks, "pool": blocks + rng.randint(1, 200),
                "block_bytes": rng.choice([2, 4, 8, 16, 18, 32]) * KIB, "op": rng.choice(["WRITE", "READ"])}
    if family == "kv":
        heads = rng.choice([1, 2, 4, 8])
        pairs = _log(rng, 1, 256)
        return {"family": "kv", "tensors": rng.choice([2, 16, 24, 48, 64, 72]), "pairs": pairs, "pool": pairs + rng.randint(0, 100),
                "tokens": rng.choice([8, 16, 16, 24]), "heads": heads, "dst_heads": heads * rng.choice([1, 2]), "dim": rng.choice([64, 96, 128]),
                "src_order": rng.choice(["NHD", "HND"]), "dst_order": rng.choice(["NHD", "HND"]), "fp8": rng.random() < 0.5}
    if family == "ep":
        ll = rng.random() < 0.5
        experts = rng.choice([4, 8, 16, 32, 64])
        return {"family": "ep", "tokens": _log(rng, 1, 256 if ll else 4096), "hidden": 512 * rng.randint(2, 14), "experts": experts,
                "topk": rng.randint(1, min(8, experts)), "low_latency": ll, "logfmt": ll and rng.random() < 0.3}
    if family == "moe":
        ll = rng.random() < 0.5
        experts = rng.choice([4, 8, 16, 32])
        return {"family": "moe", "tokens": _log(rng, 1, 256 if ll else 4096), "hidden": 512 * rng.randint(2, 8), "experts": experts,
                "topk": rng.randint(1, min(8, experts)), "low_latency": ll}
    mx = rng.random() < 0.5
    return {"family": "gemm", "groups": rng.choice([1, 3, 8, 16, 32, 40]), "rows": _log(rng, 1, 16384), "n": (256 if mx else 128) * rng.randint(1, 8),
            "k": (512 if mx else 128) * rng.randint(1, 14), "mx": mx}


# ---------------------------------------------------------------------- descriptor transfers

_agents = []


def _pair():
    """The two agents of this process, as a program keeps them for its life: one posts, the other owns the remote memory."""
    if not _agents:
        cfg = nixl_agent_config(enable_prog_thread=False, backends=["NVLINK"])
        _agents.extend((nixl_agent("cases_initiator", cfg), nixl_agent("cases_target", cfg)))
    return _agents


class _Registered:
    """Memory of both sides, registered for as long as the object lives."""

    def __init__(self, mine, theirs):
        self.a, self.b = _pair()
        self.mine, self.theirs = mine, theirs
        self.regs = [(self.a, self.a.register_memory(mine)), (self.b, self.b.register_memory(theirs))]
        self.a.add_remote_agent(self.b.get_agent_metadata())

    def release(self):
        torch.cuda.synchronize()
        for agent, reg in self.regs:
            agent.deregister_memory(reg)
        self.regs = []


def _wait(agent, handle, state):
    while state == "PROC":
        state = agent.check_xfer_state(handle)
    if state != "DONE":
        raise RuntimeError("transfer failed")


class _Xfer(_Registered):
    def __init__(self, case, seed):
        rng = np.random.default_rng(seed)
        n, size, align = case["descs"], case["bytes"], case["align"]
        lens, unit = np.full(n, size, dtype=np.int64), min(align, 16)
        if case["ragged"]:  # from an eighth of the size to the size, in whole units of up to 16 bytes
            lens = np.maximum(unit, (np.exp(rng.uniform(np.log(size / 8), np.log(size), n)) / unit).astype(np.int64) * unit)

        def place(order, gaps):
            # byte offsets of the blocks, in `order`, each at a multiple of `align`
            at, offs = 0, np.empty(n, dtype=np.int64)
            for i in order:
                at = (at + align - 1) // align * align + int(gaps[i])
                offs[i] = at
                at += int(lens[i])
            return offs, at

        gaps = rng.integers(0, 4, n) * align if case["ragged"] else np.zeros(n, dtype=np.int64)
        src_at, src_size = place(range(n), gaps)
        dst_at, _ = place(rng.permutation(n), np.zeros(n, dtype=np.int64))
        gen = torch.Generator(device="cuda").manual_seed(seed)
        src = torch.randint(0, 256, (src_size,), dtype=torch.uint8, device="cuda", generator=gen)
        dst = torch.zeros(n * (max(size, unit) + align), dtype=torch.uint8, device="cuda")  # room for the longest lengths, whatever the seed
        if case["host"]:  # the posting side's memory is pinned host memory
            if case["op"] == "WRITE":
                src = src.cpu().pin_memory()
            else:
                dst = dst.cpu().pin_memory()
        self.dst = dst
        write = case["op"] == "WRITE"
        super().__init__(src if write else dst, dst if write else src)
        # (the tensors are filled above; the handle is made once and posted again and again)
        ends = []
        for t, at in ((src, src_at), (dst, dst_at)):
            rows = np.stack([t.data_ptr() + at, lens, np.zeros(n, dtype=np.int64)], axis=1).astype(np.uint64)
            ends.append(self.a.get_xfer_descs(rows, "VRAM" if t.is_cuda else "DRAM"))
        self.handle = self.a.initialize_xfer(case["op"], ends[0 if write else 1], ends[1 if write else 0], self.b.name)

    def run(self):
        _wait(self.a, self.handle, self.a.transfer(self.handle))
        return self.dst

    def __del__(self):
        self.a.release_xfer_handle(self.handle)
        self.release()


class _Blocks(_Registered):
    def __init__(self, case, seed):
        gen = torch.Generator(device="cuda").manual_seed(seed)
        shape = (case["tensors"], case["pool"], case["block_bytes"])
        full = torch.randint(0, 256, shape, dtype=torch.uint8, device="cuda", generator=gen)
        empty = torch.zeros(shape, dtype=torch.uint8, device="cuda")
        write = case["op"] == "WRITE"
        mine, theirs = (full, empty) if write else (empty, full)
        super().__init__(mine, theirs)
        self.dst, self.op = empty, case["op"]
        self.kv = KVBlockTransfer(self.a, list(mine), self.b.name, describe_blocks(self.b, list(theirs)))
        rng = np.random.default_rng(seed)
        self.here = rng.permutation(case["pool"])[: case["blocks"]].tolist()
        self.there = rng.permutation(case["pool"])[: case["blocks"]].tolist()

    def run(self):
        self.kv.wait(self.kv.post(self.here, self.there, self.op))
        return self.dst

    def __del__(self):
        self.kv.close()
        self.release()


class _KV(_Registered):
    def __init__(self, case, seed):
        gen = torch.Generator(device="cuda").manual_seed(seed)
        n, pool, t, d = case["tensors"], case["pool"], case["tokens"], case["dim"]

        def shape(order, heads):
            return (n, pool, t, heads, d) if order == "NHD" else (n, pool, heads, t, d)

        src = torch.randn(shape(case["src_order"], case["heads"]), device="cuda", dtype=torch.bfloat16, generator=gen)
        dst = torch.zeros(shape(case["dst_order"], case["dst_heads"]), device="cuda", dtype=torch.uint8 if case["fp8"] else torch.bfloat16)
        super().__init__(src, dst)
        self.dst = dst
        size = dst[0].numel() * dst.element_size()
        self.kv = KVTransfer(self.a, list(src), KVLayout(t, case["heads"], d, case["src_order"]), self.b.name,
                             [(x.data_ptr(), size, x.get_device()) for x in dst],
                             KVLayout(t, case["dst_heads"], d, case["dst_order"], 1 if case["fp8"] else 2),
                             dst_head_offset=case["dst_heads"] - case["heads"], cast_fp8=case["fp8"], scale=16.0 if case["fp8"] else 1.0)
        self.here = torch.randperm(pool, device="cuda", generator=gen)[: case["pairs"]].int()
        self.there = torch.randperm(pool, device="cuda", generator=gen)[: case["pairs"]].int()

    def run(self):
        self.kv.post(self.here, self.there)  # in stream order; a program polls the ticket later
        return self.dst

    def __del__(self):
        torch.cuda.synchronize()
        self.kv.close()
        self.release()


# ---------------------------------------------------------------------- expert parallel

def _routing(case, seed):
    """Tokens, expert numbers and weights of a top-k router over N(0,1) logits."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.randn(case["tokens"], case["hidden"], device="cuda", dtype=torch.bfloat16, generator=gen)
    logits = torch.randn(case["tokens"], case["experts"], device="cuda", generator=gen)
    w, idx = torch.topk(torch.softmax(logits, dim=-1), case["topk"], dim=-1)
    return x, idx.contiguous(), w.float().contiguous()


def _buffer(case):
    return Buffer(0, 1, case["experts"], case["hidden"], case["tokens"], case["topk"], device=torch.device("cuda:0"),
                  low_latency_mode=case["low_latency"])


class _Ep:
    """Dispatch in bf16, experts that return what they receive, combine."""

    def __init__(self, case, seed):
        self.x, self.idx, self.w = _routing(case, seed)
        self.buf = _buffer(case)
        self.buf.connect_ranks()
        self.low_latency, self.logfmt = case["low_latency"], case["logfmt"]

    def run(self):
        if self.low_latency:
            recv, count, h, _, _ = self.buf.low_latency_dispatch(self.x, self.idx, use_fp8=False)
            out, _, _ = self.buf.low_latency_combine(recv, self.idx, self.w, h, use_logfmt=self.logfmt)
        else:
            recv, _, h = self.buf.dispatch(self.x, self.idx, use_fp8=False, topk_weights=self.w)
            out, count = self.buf.combine(recv, self.idx, self.w, h), h.recv_count
        return {"out": out, "count": count, "range": h.layout_range}


def _weights(case, seed, mx):
    """fp8 expert weights [experts, hidden, hidden] and their scales, quantised one expert at a time."""
    gen = torch.Generator(device="cuda").manual_seed(seed + 1)
    e, n, k = case.get("experts", case.get("groups")), case.get("n", case.get("hidden")), case.get("k", case.get("hidden"))
    w = torch.empty(e, n, k, dtype=torch.float8_e4m3fn, device="cuda")
    s = torch.empty(e, n // 128, k // 128, dtype=torch.uint8 if mx else torch.float32, device="cuda")
    for g in range(e):
        q, qs = (quantize_weights_ue8m0 if mx else quantize_weights)(torch.randn(1, n, k, device="cuda", generator=gen) / math.sqrt(k))
        w[g], s[g] = q[0], qs[0]
    return w, s


class _Moe:
    """Dispatch in fp8, one expert GEMM that writes where combine reads, combine."""

    def __init__(self, case, seed):
        self.x, self.idx, self.w = _routing(case, seed)
        self.low_latency, self.hidden = case["low_latency"], case["hidden"]
        self.wq, self.ws = _weights(case, seed, not self.low_latency)
        self.status = torch.zeros(1, dtype=torch.int32, device="cuda")
        self.buf = _buffer(case)
        self.buf.connect_ranks()

    def run(self):
        if self.low_latency:
            (recv, scales), count, h, _, _ = self.buf.low_latency_dispatch(self.x, self.idx, use_fp8=True)
            y = self.buf.get_next_combine_buffer(h)
            grouped_gemm_fp8(recv.view(-1, self.hidden), scales.view(-1, self.hidden // 128), self.wq, self.ws, h.expert_offsets, count,
                             out=y.view(-1, self.hidden), status=self.status)
            out, _, _ = self.buf.low_latency_combine(y, self.idx, self.w, h, zero_copy=True)
        else:
            recv, scales, h = self.buf.dispatch(self.x, self.idx, use_ue8m0=True, topk_weights=self.w)
            y = self.buf.get_next_combine_buffer(h)
            grouped_gemm_mxfp8(recv, scales, self.wq, self.ws, h.expert_offsets, h.recv_count, out=y, status=self.status)
            out, count = self.buf.combine(y, self.idx, self.w, h), h.recv_count
        return {"out": out, "count": count, "status": self.status}


def _quantise_rows(x, mx):
    """1 x 128 e4m3 blocks of the rows of x: codes and fp32 scales (powers of two with `mx`)."""
    g = x.float().view(x.shape[0], -1, 128)
    amax = g.abs().amax(dim=2).clamp(min=1e-4)
    full = torch.full_like(amax, 448.0)
    if mx:
        ex = torch.ceil(torch.log2(amax / full))
        scale, inv = torch.exp2(ex), torch.exp2(-ex)
    else:
        scale, inv = amax / full, full / amax
    return (g * inv.unsqueeze(2)).to(torch.float8_e4m3fn).view(x.shape), scale


class _Gemm:
    def __init__(self, case, seed):
        gen = torch.Generator(device="cuda").manual_seed(seed)
        rows, groups = case["rows"], case["groups"]
        # Some experts are asked for more often than others, and a few hardly at all.
        share = torch.exp(0.5 * torch.randn(groups, device="cuda", generator=gen))
        share[0] = 0 if groups > 2 else share[0]
        counts = torch.bincount(torch.multinomial(share, rows, replacement=True, generator=gen), minlength=groups)
        self.count = counts.int()
        self.start = (torch.cumsum(counts, 0) - counts).int()
        x = torch.randn(rows, case["k"], device="cuda", dtype=torch.bfloat16, generator=gen)
        self.mx = case["mx"]
        self.a, self.sa = _quantise_rows(x, self.mx)
        if self.mx:
            self.sa = to_ue8m0(self.sa)
        self.w, self.sw = _weights(case, seed, self.mx)
        self.status = torch.zeros(1, dtype=torch.int32, device="cuda")

    def run(self):
        gemm = grouped_gemm_mxfp8 if self.mx else grouped_gemm_fp8
        out = gemm(self.a, self.sa, self.w, self.sw, self.start, self.count, status=self.status)
        return {"out": out, "status": self.status}


# ---------------------------------------------------------------------- the interface

_FAMILIES = {"xfer": _Xfer, "blocks": _Blocks, "kv": _KV, "ep": _Ep, "moe": _Moe, "gemm": _Gemm}


def prepare(case, seed):
    return _FAMILIES[case["family"]](case, seed)


def run(state):
    return state.run()


def work(case):
    f = case["family"]
    if f == "xfer":
        # ragged lengths are log-uniform between size / 8 and size: their mean is (1 - 1/8) / ln 8 of the size
        mean = case["bytes"] * (0.875 / math.log(8) if case["ragged"] else 1.0)
        return {"bytes": 2 * case["descs"] * max(1.0, mean), "flops": 0}
    if f == "blocks":
        return {"bytes": 2 * case["tensors"] * case["blocks"] * case["block_bytes"], "flops": 0}
    if f == "kv":
        elems = case["tensors"] * case["pairs"] * case["tokens"] * case["heads"] * case["dim"]
        return {"bytes": elems * (3 if case["fp8"] else 4), "flops": 0}
    if f == "gemm":
        rows, n, k, g = case["rows"], case["n"], case["k"], min(case["groups"], case["rows"])
        return {"bytes": rows * k + g * n * k + 2 * rows * n, "flops": 2 * rows * n * k}
    t, h, copies = case["tokens"], case["hidden"], case["tokens"] * case["topk"]
    if f == "ep":  # tokens in, copies out; copies in, tokens out
        return {"bytes": 2 * h * (t + copies) * 2, "flops": 2 * copies * h}
    experts = min(case["experts"], copies)
    return {"bytes": 2 * h * t + h * copies + (h * copies + experts * h * h + 2 * h * copies) + 2 * h * copies + 2 * h * t,
            "flops": 2 * copies * h * h + 2 * copies * h}


def tolerance(case):
    f = case["family"]
    if f in ("xfer", "blocks", "kv"):
        return "exact"  # bytes that are moved, and fp8 codes of single values
    # bf16 results of fp32 sums: in another order of the sum a result that lies near the middle of two bf16 values
    # becomes its neighbour (one step is up to 2^-7 of the value); an intermediate row may do so too before it is added up.
    # Measured against 64 bits: 1.7e-3 with one rounding to bf16, 2.3e-3 where the experts' rows are rounded too.
    if f == "ep" and case["logfmt"]:
        return {"rel": 1e-2, "max": 0.06}  # rows travel as 9-bit codes
    return {"rel": 7e-3, "max": 0.03}


def exact(case, seed):
    f = case["family"]
    if f == "ep":
        x, idx, w = _routing(case, seed)
        return {"out": x.double() * w.double().sum(dim=1, keepdim=True), "count": None, "range": None}
    if f == "gemm":
        s = _Gemm(case, seed)
        a = _dequantise_rows(s.a, s.sa, s.mx)
        out = torch.empty(case["rows"], case["n"], dtype=torch.float64, device="cuda")
        at = 0
        for g, c in enumerate(s.count.tolist()):
            out[at : at + c] = a[at : at + c] @ _dequantise_block(s.w[g], s.sw[g], s.mx).t()
            at += c
        return {"out": out, "status": None}
    if f == "moe":
        x, idx, w = _routing(case, seed)
        mx = not case["low_latency"]
        wq, ws = _weights(case, seed, mx)
        a = _dequantise_rows(*_quantise_rows(x, mx), False)
        out = torch.zeros(x.shape, dtype=torch.float64, device="cuda")
        for e in range(case["experts"]):
            t, k = torch.nonzero(idx == e, as_tuple=True)
            out.index_add_(0, t, (a[t] @ _dequantise_block(wq[e], ws[e], mx).t()) * w[t, k].double().unsqueeze(1))
        return {"out": out, "count": None, "status": None}
    return None


def _scales(s, mx):
    return torch.exp2(s.double() - 127.0) if mx else s.double()


def _dequantise_rows(q, s, mx):
    return (q.double().view(q.shape[0], -1, 128) * _scales(s, mx).unsqueeze(2)).view(q.shape)


def _dequantise_block(q, s, mx):
    n, k = q.shape
    return (q.double().view(n // 128, 128, k // 128, 128) * _scales(s, mx)[:, None, :, None]).view(n, k)
