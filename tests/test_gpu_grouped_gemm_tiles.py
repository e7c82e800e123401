"""The CTA-pair grouped GEMMs at the row counts where their tiles change: the fp32-scale kernel runs a tile with at most 128
rows left as M = 128, the block-scaled one splits an expert's rows into equal tiles of at most 256, rounded up to 32.  Rows that
belong to no expert must stay as they were."""
import pytest
import torch

from nixl_b200.ops import from_ue8m0, grouped_gemm_fp8, grouped_gemm_mxfp8, to_ue8m0

pytestmark = pytest.mark.gpu

_COUNTS = [
    [1, 63, 64, 65],
    [127, 128, 129, 0, 191],
    [255, 256, 257, 31, 32, 33],
    [384, 385, 512, 513, 2],
]


def _inputs(counts, N, K, seed):
    dev = torch.device("cuda:0")
    g = torch.Generator(device=dev).manual_seed(seed)
    starts, run = [], 3
    for c in counts:
        starts.append(run)
        run += c + 2
    a = (torch.randn(run, K, device=dev, generator=g) * 60).to(torch.float8_e4m3fn)
    w = (torch.randn(len(counts), N, K, device=dev, generator=g) * 60).to(torch.float8_e4m3fn)
    rs = torch.tensor(starts, dtype=torch.int32, device=dev)
    rc = torch.tensor(counts, dtype=torch.int32, device=dev)
    # scales that differ per row, step and weight block, powers of two so that both kernels can take them
    sa = torch.exp2(torch.randint(-9, -3, (run, K // 128), device=dev, generator=g).float())
    sw = torch.exp2(torch.randint(-9, -3, (len(counts), N // 128, K // 128), device=dev, generator=g).float())
    return a, sa, w, sw, rs, rc


def _check(out, a, sa, w, sw, rs, rc, K):
    seen = torch.zeros(a.shape[0], dtype=torch.bool, device=a.device)
    af = (a.double().view(a.shape[0], -1, 128) * sa.double().unsqueeze(2)).view(a.shape)
    for g, (s, c) in enumerate(zip(rs.tolist(), rc.tolist())):
        if c == 0:
            continue
        wf = (w[g].double().view(w.shape[1] // 128, 128, -1, 128) * sw[g].double()[:, None, :, None]).view(w.shape[1], -1)
        want = af[s : s + c] @ wf.t()
        # one rounding to bf16 (half a step: 2^-9 of the value, or less), K additions in fp32 of terms whose magnitudes sum up to `mass`
        mass = af[s : s + c].abs() @ wf.abs().t()
        bound = want.abs() * 2.0**-8 + mass * (K * 2.0**-24)
        err = (out[s : s + c].double() - want).abs()
        assert bool((err <= bound).all()), (g, c, float((err / bound).max()))
        seen[s : s + c] = True
    assert bool((out[~seen] == 5.0).all())


@pytest.mark.parametrize("counts", _COUNTS)
@pytest.mark.parametrize("N,K", [(256, 128), (768, 640), (512, 4224)])
def test_fp32_scales(counts, N, K):
    a, sa, w, sw, rs, rc = _inputs(counts, N, K, 1)
    out = torch.full((a.shape[0], N), 5.0, dtype=torch.bfloat16, device=a.device)
    grouped_gemm_fp8(a, sa, w, sw, rs, rc, out=out, tile_mode=2)
    torch.cuda.synchronize()
    assert int(out._nixl_status.item()) == 0
    _check(out, a, sa, w, sw, rs, rc, K)


@pytest.mark.parametrize("counts", _COUNTS)
@pytest.mark.parametrize("N,K", [(256, 512), (768, 1536), (512, 4608)])  # one scale group, part of one, more than one
def test_block_scales(counts, N, K):
    a, sa, w, sw, rs, rc = _inputs(counts, N, K, 2)
    out = torch.full((a.shape[0], N), 5.0, dtype=torch.bfloat16, device=a.device)
    sab, swb = to_ue8m0(sa), to_ue8m0(sw)
    assert torch.equal(from_ue8m0(sab), sa)
    grouped_gemm_mxfp8(a, sab, w, swb, rs, rc, out=out)
    torch.cuda.synchronize()
    assert int(out._nixl_status.item()) == 0
    _check(out, a, sa, w, sw, rs, rc, K)


@pytest.mark.parametrize("groups,rows,N", [(2, 256, 256), (2, 257, 2560), (4, 300, 2304), (1, 2048, 256)])
def test_either_side_of_the_tile_shape_rule(groups, rows, N):
    K = 512
    a, sa, w, sw, rs, rc = _inputs([rows] * groups, N, K, 3)
    out = torch.full((a.shape[0], N), 5.0, dtype=torch.bfloat16, device=a.device)
    grouped_gemm_fp8(a, sa, w, sw, rs, rc, out=out)
    torch.cuda.synchronize()
    _check(out, a, sa, w, sw, rs, rc, K)


@pytest.mark.parametrize("counts", [[1, 32], [33, 7, 0], [64, 64, 64], [65, 1], [128, 32, 33], [129, 31, 256]])  # the fullest expert sets the stages
@pytest.mark.parametrize("N,K", [(128, 128), (384, 1664)])
def test_single_cta_tiles(counts, N, K):
    a, sa, w, sw, rs, rc = _inputs(counts, N, K, 4)
    out = torch.full((a.shape[0], N), 5.0, dtype=torch.bfloat16, device=a.device)
    grouped_gemm_fp8(a, sa, w, sw, rs, rc, out=out, tile_mode=1)
    torch.cuda.synchronize()
    assert int(out._nixl_status.item()) == 0
    _check(out, a, sa, w, sw, rs, rc, K)
