"""The grouped GEMMs with several tiles of different sizes per CTA or CTA pair: what the roles carry from tile to tile (ring
positions, parities, scale groups, the accumulator's hand-back).  `grid` holds the launch to a few CTAs; with the default
grid the shapes of test_gpu_grouped_gemm_tiles.py give a pair one tile at most."""
import pytest
import torch

from nixl_b200.ops import grouped_gemm_fp8, grouped_gemm_mxfp8, to_ue8m0
from test_gpu_grouped_gemm_tiles import _check, _inputs

pytestmark = pytest.mark.gpu

_MIXED = [1, 300, 32, 0, 129, 513, 64, 255, 257]  # tiles of 32 to 256 tokens in turn


def _run(gemm, counts, N, K, grid, seed, mx=False, **kw):
    a, sa, w, sw, rs, rc = _inputs(counts, N, K, seed)
    for _ in range(3):  # the bound of _check leaves no room for a tile that was overwritten while it was read
        out = torch.full((a.shape[0], N), 5.0, dtype=torch.bfloat16, device=a.device)
        gemm(a, to_ue8m0(sa) if mx else sa, w, to_ue8m0(sw) if mx else sw, rs, rc, out=out, grid=grid, **kw)
        torch.cuda.synchronize()
        assert int(out._nixl_status.item()) == 0
        _check(out, a, sa, w, sw, rs, rc, K)


@pytest.mark.parametrize("grid", [2, 4, 6])
@pytest.mark.parametrize("N,K", [(512, 1024), (768, 1536), (256, 4608), (512, 8704)])  # 2, 3, 9 and 17 chunks of scales: one to three groups
def test_block_scales_that_one_thread_copies_and_the_other_uses(grid, N, K):
    _run(grouped_gemm_mxfp8, _MIXED, N, K, grid, 11, mx=True)


@pytest.mark.parametrize("grid", [2, 4, 6])
@pytest.mark.parametrize("N", [256, 1024])
def test_block_scales_with_one_chunk_per_tile(grid, N):
    """K = 512: the two issuing threads take whole tiles in turn, and only the wait for the accumulator keeps them apart."""
    _run(grouped_gemm_mxfp8, _MIXED, N, 512, grid, 12, mx=True)
    _run(grouped_gemm_mxfp8, [256] * 24, N, 512, grid, 13, mx=True)


@pytest.mark.parametrize("grid", [2, 4, 6])
@pytest.mark.parametrize("N,K", [(512, 128), (768, 640), (256, 1408)])  # 1, 5 and 11 steps: every tile starts in another TMEM slot pair
def test_fp32_scales_full_and_tail_tiles_in_turn(grid, N, K):
    _run(grouped_gemm_fp8, _MIXED, N, K, grid, 14, tile_mode=2)


@pytest.mark.parametrize("grid", [1, 2, 3])
@pytest.mark.parametrize("counts", [[1, 32, 7, 0, 30] * 3, [33, 64, 2, 50] * 3, _MIXED])  # stages for 32, 64 and 128 rows
@pytest.mark.parametrize("N,K", [(256, 128), (384, 1664)])
def test_single_ctas_with_each_depth_of_the_ring(grid, counts, N, K):
    _run(grouped_gemm_fp8, counts, N, K, grid, 15, tile_mode=1)
