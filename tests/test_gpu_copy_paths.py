"""The descriptor copy kernels at the sizes and alignments where they can go wrong: every relative alignment of source and
destination, lengths around the vector, warp and chunk sizes, descriptor tables that ride in the launch parameters and
that do not, chunks for warps and for whole CTAs.  Bytes outside the destinations must stay as they were."""
import numpy as np
import pytest
import torch

from nixl_b200 import nixl_agent, nixl_agent_config

pytestmark = pytest.mark.gpu

_LENGTHS = [1, 15, 16, 31, 33, 63, 64, 65, 94, 511, 2047, 2048, 2049, 4095, 4096, 4097, 4111, 8193, 32768, 32801, 65537, 131103]


def _move(tag, lens, src_at, dst_at, params):
    cfg = nixl_agent_config(enable_prog_thread=False, backends=[])
    a, b = nixl_agent(f"{tag}_a", cfg), nixl_agent(f"{tag}_b", cfg)
    params = {"coalesce": "false", "proxy": "false", **params}
    a.create_backend("NVLINK", params)
    b.create_backend("NVLINK", params)
    lens, src_at, dst_at = (np.asarray(v, dtype=np.int64) for v in (lens, src_at, dst_at))
    src = torch.randint(0, 256, (int((src_at + lens).max()) + 64,), dtype=torch.uint8, device="cuda:0")
    dst = torch.randint(0, 256, (int((dst_at + lens).max()) + 64,), dtype=torch.uint8, device="cuda:0")
    want = dst.cpu().numpy()
    from_ = src.cpu().numpy()
    for n, s, d in zip(lens, src_at, dst_at):
        want[d : d + n] = from_[s : s + n]
    ra, rb = a.register_memory(src), b.register_memory(dst)
    a.add_remote_agent(b.get_agent_metadata())
    ends = [a.get_xfer_descs(np.stack([t.data_ptr() + at, lens, np.zeros_like(lens)], axis=1).astype(np.uint64), "VRAM") for t, at in ((src, src_at), (dst, dst_at))]
    h = a.initialize_xfer("WRITE", ends[0], ends[1], b.name)
    state = a.transfer(h)
    while state == "PROC":
        state = a.check_xfer_state(h)
    assert state == "DONE"
    torch.cuda.synchronize()
    got = dst.cpu().numpy()
    bad = np.nonzero(got != want)[0]
    assert bad.size == 0, (bad.size, bad[:8])
    a.release_xfer_handle(h)
    a.deregister_memory(ra)
    b.deregister_memory(rb)


def _place(lens, offs, pitch=64):
    at, out = 0, []
    for n, o in zip(lens, offs):
        out.append(at + int(o))
        at += -(-(int(n) + int(o) + 1) // pitch) * pitch + pitch
    return out


# chunk_shift 0: the backend chooses (warps here); 12: short chunks for warps; 16: chunks for CTAs
@pytest.mark.parametrize("shift", ["0", "12", "16"])
def test_every_relative_alignment(shift):
    lens, so, do = [], [], []
    for s in range(0, 32):
        for d in (0, 1, 7, 16, 29):
            lens.append(_LENGTHS[(5 * s + d) % len(_LENGTHS)])
            so.append(s)
            do.append(d)
    _move(f"cpa{shift}", lens, _place(lens, so), _place(lens, do), {"chunk_shift": shift})


@pytest.mark.parametrize("shift", ["0", "16"])
@pytest.mark.parametrize("dst_off", [0, 3, 16])
def test_lengths_around_vectors_warps_and_chunks(shift, dst_off):
    for lens in (_LENGTHS, _LENGTHS * 3):  # inside the launch parameters (22 descriptors) and in a table (66)
        _move(f"cpl{shift}_{dst_off}_{len(lens)}", lens, _place(lens, [0] * len(lens)), _place(lens, [dst_off] * len(lens)), {"chunk_shift": shift})


@pytest.mark.parametrize("n", [1, 31, 32, 33, 1024, 1025, 2500])  # around the widths of the warp-wide search
@pytest.mark.parametrize("uniform", [True, False])
def test_descriptor_search(n, uniform):
    rng = np.random.default_rng(n)
    lens = np.full(n, 8192) if uniform else rng.integers(1, 20000, n)
    src_at = _place(lens, np.zeros(n, dtype=int))
    dst_at = np.array(_place(lens, np.zeros(n, dtype=int)))
    _move(f"cps{n}_{uniform}", lens, src_at, dst_at, {})


def test_either_side_of_the_request_size_rule():
    for extra in (0, 4096):  # 64 MiB go to warps, more to CTAs
        size = (16 << 20) + extra // 4
        at = [i * (size + 256) for i in range(4)]
        _move(f"cpr{extra}", [size] * 4, at, at[::-1], {})


@pytest.mark.parametrize("op", ["WRITE", "READ"])
@pytest.mark.parametrize("pinned", [True, False])
@pytest.mark.parametrize(
    "lens",
    [[4096], [64 << 10], [(64 << 10) + 1], [1, 63, 4097, 70000], [(4 << 20) - 1, 4 << 20, 5, (4 << 20) + 3], [333] * 300],
)
def test_host_memory_either_side_of_the_copy_engine_rule(op, pinned, lens):
    """Host memory pinned by its owner (short pieces by the kernel, long or single ones by copies) or by the registration."""
    tag = f"cph{op}{int(pinned)}{len(lens)}_{lens[0]}"
    cfg = nixl_agent_config(enable_prog_thread=False, backends=["NVLINK"])
    a, b = nixl_agent(f"{tag}_a", cfg), nixl_agent(f"{tag}_b", cfg)
    lens = np.asarray(lens, dtype=np.int64)
    at = [np.array(_place(lens, [o] * len(lens))) for o in (3, 16)]
    size = [int((x + lens).max()) + 64 for x in at]
    host = torch.randint(0, 256, (size[0],), dtype=torch.uint8)
    host = host.pin_memory() if pinned else host
    dev = torch.randint(0, 256, (size[1],), dtype=torch.uint8, device="cuda:0")
    want_h, want_d = host.numpy().copy(), dev.cpu().numpy()
    for n, h, d in zip(lens, *at):
        if op == "WRITE":
            want_d[d : d + n] = want_h[h : h + n]
        else:
            want_h[h : h + n] = want_d[d : d + n]
    ra, rb = a.register_memory(host), b.register_memory(dev)
    a.add_remote_agent(b.get_agent_metadata())
    ends = [a.get_xfer_descs(np.stack([t.data_ptr() + x, lens, np.zeros_like(lens)], axis=1).astype(np.uint64), m) for t, x, m in ((host, at[0], "DRAM"), (dev, at[1], "VRAM"))]
    h = a.initialize_xfer(op, ends[0], ends[1], b.name, b"there")
    for _ in range(2):
        state = a.transfer(h)
        while state == "PROC":
            state = a.check_xfer_state(h)
        assert state == "DONE"
    torch.cuda.synchronize()
    assert np.array_equal(host.numpy(), want_h) and np.array_equal(dev.cpu().numpy(), want_d)
    seen = 0
    for _ in range(100000):
        seen += len(b.get_new_notifs().get(a.name, []))
        if seen == 2:
            break
    assert seen == 2  # every post delivers its message
    a.release_xfer_handle(h)
    a.deregister_memory(ra)
    b.deregister_memory(rb)
