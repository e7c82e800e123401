// Internal interface between the grouped-GEMM kernels and their common launcher.
#ifndef NIXL_B200_GROUPED_GEMM_INTERNAL_H
#define NIXL_B200_GROUPED_GEMM_INTERNAL_H

#include <cuda.h>
#include <cuda_runtime.h>

#include "kernels/nixl_kernels.h"
#ifdef __CUDACC__
#include "kernels/tcgen05_ptx.cuh"
#endif

namespace nixl_gemm {

enum : int { GEMM_ERR_TIMEOUT = 1, GEMM_ERR_ARRIVAL = 2 };
constexpr int kMaxGroups = 512;

// 2-D tensor map over a row-major [rows, k] byte matrix, boxes of box_rows x 128 bytes, 128-byte swizzle.
bool makeTileMap(CUtensorMap *map, const void *base, uint64_t rows, uint64_t k, uint32_t box_rows = 128);
// The same matrix as [k / 128][rows][128 bytes], boxes of two neighbouring 128-byte columns x 128 rows: they land one behind the
// other, each as a box of the map above would.  A second column past the end of k is filled with zeros.
bool makePairMap(CUtensorMap *map, const void *base, uint64_t rows, uint64_t k);

// 256 x 256 tiles computed by CTA pairs (tcgen05 cta_group::2).  Same contract as the
// single-CTA kernel; N must be a multiple of 256.  The maps of A have boxes of 128 and 64 rows, that of W 128.
cudaError_t launchPairKernel(const CUtensorMap &mapA, const CUtensorMap &mapA64, const CUtensorMap &mapW, const NixlGroupedGemmParams &p, cudaStream_t stream);

// Tiles of 256 columns x up to 256 tokens with power-of-two block scales applied by the tensor core (kind::mxf8f6f4.block_scale):
// p.scale_a / p.scale_w point at exponent bytes (uint8 [a_rows][K/128] and [groups][N/128][K/128]);
// K must be a multiple of 512, N of 256; no dispatch overlap.  The maps of the tokens have boxes of 128, 32 and 64 rows.
// mapW2 is that of makePairMap.
cudaError_t launchMxPairKernel(const CUtensorMap &mapT, const CUtensorMap &mapT32, const CUtensorMap &mapT64, const CUtensorMap &mapW, const CUtensorMap &mapW2,
                               const NixlGroupedGemmParams &p, cudaStream_t stream);

#ifdef __CUDACC__
// The tile table of a launch, built by one whole warp, 32 groups at a time: prefix[g] tiles come before group g, each of whose
// tilesOf(rows) row tiles has n_tiles columns of tiles.  One thread that walked the groups took a load's latency for each.
template<class TilesOf>
__device__ __forceinline__ void buildTileTable(const NixlGroupedGemmParams &p, int n_tiles, TilesOf tilesOf, int *prefix, int *rowStart, int *rowCount, int &most) {
    const int lane = threadIdx.x & 31;
    int run = 0, top = 0;
    for (int g0 = 0; g0 < p.groups; g0 += 32) {
        const int g = g0 + lane;
        const int count = g < p.groups ? p.row_count[g] : 0, start = g < p.groups ? p.row_start[g] : 0;
        const int here = tilesOf(count) * n_tiles;
        int upto = here;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int below = __shfl_up_sync(0xffffffffu, upto, o);
            if (lane >= o) upto += below;
        }
        if (g < p.groups) {
            prefix[g] = run + upto - here;
            rowStart[g] = start;
            rowCount[g] = count;
        }
        run += __shfl_sync(0xffffffffu, upto, 31);
        top = max(top, count);
    }
    if (lane == 0) prefix[p.groups] = run;
    most = __reduce_max_sync(0xffffffffu, top);
}
// Waits (bounded) until the rows [lo, hi) of group g have arrived: rows of an expert are ordered by source rank, so for the
// arrival flags of the sources whose rows intersect the range.  On expiry the host sees the status bit and the kernel
// computes on what is there.
__device__ __forceinline__ void waitArrivals(const NixlGroupedGemmParams &p, int g, int lo, int hi) {
    int first = 0;
    for (int r = 0; r < p.ranks; ++r) {
        const int c = p.counts[static_cast<long long>(r) * p.experts_total + p.expert_base + g];
        if (c > 0 && first < hi && first + c > lo) {
            const uint64_t *flag = p.disp_flag + static_cast<long long>(g) * p.ranks + r;
            uint64_t t0 = 0;
            unsigned spins = 0;
            while (nixl_tc::ldAcquireSys(flag) < p.epoch) {
                if ((++spins & 63u) == 0) {
                    const uint64_t now = nixl_tc::nowNs();
                    if (t0 == 0) t0 = now;
                    else if (now - t0 > p.timeout_ns) {
                        atomicOr(p.status, GEMM_ERR_ARRIVAL);
                        break;
                    }
                }
            }
        }
        first += c;
    }
}
// A scale, or four exponent bytes.  Not through the read-only path, which is for data that nobody writes while the kernel runs: the
// kernel in front writes the scales of A, and may write those of W, while this one sets itself up.  `fresh`: a dispatch writes them
// while this kernel's main loop runs, so L1 may hold lines from before some row's arrival.
__device__ __forceinline__ float ldScale(const float *s, bool fresh) {
    float f;
    if (fresh) asm volatile("ld.global.cg.f32 %0, [%1];" : "=f"(f) : "l"(s));
    else asm volatile("ld.global.f32 %0, [%1];" : "=f"(f) : "l"(s));
    return f;
}
__device__ __forceinline__ uint32_t ldExponents(const uint32_t *s) {
    uint32_t v;
    asm volatile("ld.global.u32 %0, [%1];" : "=r"(v) : "l"(s));
    return v;
}
// A row's scales of the four steps from ks on, in one load where they start at a multiple of 16 bytes.  The lanes of a warp read 32
// rows, that is 32 lines, and each line costs a cycle of the memory that TMA and MMA work on too.
__device__ __forceinline__ float4 ldScales4(const float *row, int ks, int k_steps, bool fresh) {
    const float *s = row + ks;
    float4 f;
    if (ks + 4 <= k_steps && (reinterpret_cast<uintptr_t>(s) & 15) == 0) {
        if (fresh) asm volatile("ld.global.cg.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(f.x), "=f"(f.y), "=f"(f.z), "=f"(f.w) : "l"(s));
        else asm volatile("ld.global.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(f.x), "=f"(f.y), "=f"(f.z), "=f"(f.w) : "l"(s));
        return f;
    }
    f.x = ks < k_steps ? ldScale(s, fresh) : 0.f;
    f.y = ks + 1 < k_steps ? ldScale(s + 1, fresh) : 0.f;
    f.z = ks + 2 < k_steps ? ldScale(s + 2, fresh) : 0.f;
    f.w = ks + 3 < k_steps ? ldScale(s + 3, fresh) : 0.f;
    return f;
}
#endif

} // namespace nixl_gemm

#endif
