// Grouped expert GEMM on 5th-generation tensor cores, optionally fed by EP dispatch arrivals.
//
//   D[rows of expert g, :] = dequant(A[rows, K]) x dequant(W[g, N, K])^T        (bf16 out)
//   A: e4m3, one fp32 scale per row per 128 channels (what EP dispatch delivers)
//   W: e4m3, one fp32 scale per 128 x 128 block
//
// sm_100a only.  One persistent CTA per SM, 384 threads, warp-specialised:
//   warp 0  TMA producer   cp.async.bulk.tensor (128-byte swizzle) of two 128-channel steps at a time into a shared-memory ring
//                          of 5, 4 or 3 stages: one box of 128 W rows x 256 channels, two of 32, 64 or 128 A rows x 128
//   warp 1  MMA issuer     4 x tcgen05.mma.kind::f8f6f4 (M128 N128 K32) per step into one of four
//                          TMEM accumulators (128 lanes x 128 fp32 columns each: all 512 columns).
//                          It polls one barrier per stage, with a non-blocking test issued behind
//                          the previous stage's MMAs (barrier instructions in front of the MMAs
//                          delay them by hundreds of cycles)
//   warp 2  TMEM allocator
//   warp 3  slot watcher   forwards "accumulators free again" into the stage's full[] barrier, so
//                          that barrier alone tells the issuer that a stage may go
//   warps 4-11 promotion + epilogue (two warps per TMEM lane quarter, 64 columns each):
//                          tcgen05.ld the step's partial sums, multiply by
//                          scaleA[row, step] * scaleW[g, n-block, step], accumulate in registers
//                          (the per-128-channel scales cannot be folded into the MMA), finally
//                          store bf16.  Four accumulators keep the MMA pipe fed across the
//                          commit -> wait -> load -> release round trip of each step.
// TMA loads read this GPU's own memory only and use no cluster multicast.  When `disp_flag` is
// given, the producer waits (bounded) for the per-(expert, source rank) arrival flags raised by
// ep_kernels.cu before it loads rows that those sources wrote: dispatch and GEMM overlap tile by
// tile instead of being separated by a receive phase.
//
// The reference has no GEMM (it moves tokens only); this kernel is the "dispatch fused into a
// tcgen05/TMEM grouped expert GEMM" variant of the EP path.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cstdio>
#include <mutex>

#include "kernels/nixl_kernels.h"
#include "kernels/grouped_gemm_internal.h"
#include "kernels/programmatic_launch.cuh"
#include "kernels/tcgen05_ptx.cuh"

namespace {

using namespace nixl_tc;

constexpr int BM = 128, BN = 128, BK = 128; // tile; BK is also the scale granularity
constexpr int kRingBytes = 200 * 1024;
constexpr int kMaxStages = 5;
constexpr int kTurned = 64;                // most rows of a tile whose operands are swapped
constexpr int kStageSteps = 2;             // 128-channel steps per stage (the last one of an odd K has one)
constexpr int kThreads = 384;              // 4 role warps + 8 promotion warps
constexpr int kTileBytes = BM * BK;         // 16 KiB (fp8)
constexpr int kTailBytes = kTileBytes - 32 * BK; // an MMA with A on its M side reads 128 A rows, also of a last stage that has room for 32
constexpr int kAccBufs = 4;                 // TMEM accumulators in flight (4 x 128 columns = all of TMEM)
constexpr int kTmemCols = kAccBufs * BN;

using nixl_gemm::GEMM_ERR_ARRIVAL;
using nixl_gemm::GEMM_ERR_TIMEOUT;
using nixl_gemm::kMaxGroups;
using nixl_gemm::ldScales4;
using nixl_gemm::waitArrivals;

struct Shared {
    uint64_t full[kMaxStages];
    uint64_t empty[kMaxStages];
    uint64_t tmemFull[kAccBufs];
    uint64_t tmemEmpty[kAccBufs];
    uint32_t tmemBase;
    int abort;
    alignas(16) float scales[8][2][32]; // of the promotion warps (swapped operands)
    int aRows;                      // A rows a stage has room for: 32, 64 or 128
    int tilePrefix[kMaxGroups + 1]; // tiles before group g
    int rowStart[kMaxGroups];
    int rowCount[kMaxGroups];
};

// Instruction descriptor: D fp32, A and B e4m3, both K-major, M = 128, N = n.
__device__ __forceinline__ constexpr uint32_t instrDesc(int n) {
    return (1u << 4) | (0u << 7) | (0u << 10) | (0u << 15) | (0u << 16) | (static_cast<uint32_t>(n >> 3) << 17) |
        (static_cast<uint32_t>(BM >> 4) << 24);
}

// The first of a stage's two steps: its four MMAs and the commit of its accumulator.
__device__ __forceinline__ void issueFirstStep(uint32_t tmem_d, uint64_t da, uint64_t dw, uint32_t idesc, uint32_t bar_tmem_full) {
    asm volatile(
        "{\n"
        " .reg .pred pacc, pnew;\n"
        " setp.ne.b32 pacc, %5, 0;\n"
        " setp.eq.b32 pnew, %5, 0;\n"
        " tcgen05.mma.cta_group::1.kind::f8f6f4 [%0], %1, %2, %3, {%6, %6, %6, %6}, pnew;\n"
        " add.u64 %1, %1, 2;\n add.u64 %2, %2, 2;\n"
        " tcgen05.mma.cta_group::1.kind::f8f6f4 [%0], %1, %2, %3, {%6, %6, %6, %6}, pacc;\n"
        " add.u64 %1, %1, 2;\n add.u64 %2, %2, 2;\n"
        " tcgen05.mma.cta_group::1.kind::f8f6f4 [%0], %1, %2, %3, {%6, %6, %6, %6}, pacc;\n"
        " add.u64 %1, %1, 2;\n add.u64 %2, %2, 2;\n"
        " tcgen05.mma.cta_group::1.kind::f8f6f4 [%0], %1, %2, %3, {%6, %6, %6, %6}, pacc;\n"
        " tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%4];\n"
        "}\n"
        : "+r"(tmem_d), "+l"(da), "+l"(dw)
        : "r"(idesc), "r"(bar_tmem_full), "r"(1u), "r"(0u)
        : "memory");
}

// One 128-channel step of the issuer as a single instruction sequence: four MMAs, the two
// commits, then a non-blocking test of the next stage's barrier.  Barrier instructions in front of
// the MMAs delay them by a few hundred cycles each, so the stage's only poll sits behind them.
__device__ __forceinline__ void issueStep(uint32_t tmem_d, uint64_t da, uint64_t dw, uint32_t idesc, uint32_t bar_tmem_full, uint32_t bar_stage_empty,
                                          uint32_t peek_bar, uint32_t peek_par, uint32_t &ready_next) {
    asm volatile(
        "{\n"
        " .reg .pred pf, pacc, pnew;\n"
        " setp.ne.b32 pacc, %9, 0;\n"
        " setp.eq.b32 pnew, %9, 0;\n"
        " tcgen05.mma.cta_group::1.kind::f8f6f4 [%1], %2, %3, %4, {%10, %10, %10, %10}, pnew;\n"
        " add.u64 %2, %2, 2;\n add.u64 %3, %3, 2;\n"
        " tcgen05.mma.cta_group::1.kind::f8f6f4 [%1], %2, %3, %4, {%10, %10, %10, %10}, pacc;\n"
        " add.u64 %2, %2, 2;\n add.u64 %3, %3, 2;\n"
        " tcgen05.mma.cta_group::1.kind::f8f6f4 [%1], %2, %3, %4, {%10, %10, %10, %10}, pacc;\n"
        " add.u64 %2, %2, 2;\n add.u64 %3, %3, 2;\n"
        " tcgen05.mma.cta_group::1.kind::f8f6f4 [%1], %2, %3, %4, {%10, %10, %10, %10}, pacc;\n"
        " tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%6];\n"
        " tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%5];\n"
        " mbarrier.test_wait.parity.shared::cta.b64 pf, [%7], %8;\n"
        " selp.u32 %0, 1, 0, pf;\n"
        "}\n"
        : "=r"(ready_next), "+r"(tmem_d), "+l"(da), "+l"(dw)
        : "r"(idesc), "r"(bar_tmem_full), "r"(bar_stage_empty), "r"(peek_bar), "r"(peek_par), "r"(1u), "r"(0u)
        : "memory");
}

// Rows of the one TMA box that fetches A for a tile with `rows` rows.  One box, not several small ones: each TMA
// instruction of a step costs its issuing thread more than the rows it may save (32 experts, 32 rows each, 2048 x 7168: one
// box of 32 92 us, two of 16 101 us).
__device__ __forceinline__ int aBoxRows(int rows) { return rows <= 32 ? 32 : rows <= 64 ? 64 : BM; }
__device__ __forceinline__ int rowTiles(int rows) { return (rows + BM - 1) / BM; }

// Promotion and store of one tile whose operands are swapped (see groupedGemmKernel): this thread's TMEM lane is column
// `lane` of the warp's 32 columns of D, the accumulator's columns are the rows of A, kCols of them this warp's.  A row's scale is loaded
// by the lane of its number and read by all from the warp's own two rows of shared memory, four at a time (shuffles, one per row and
// step, took as long as HBM took for W).  Steps take the two rows in turn; a tile's first step may take the one that the last step of
// the tile before was read from (an odd number of steps), so the warp meets in between.  False when another role gave up.
template<int kCols>
__device__ __forceinline__ bool promoteSwapped(Shared &sh, const float *sa_row, bool valid, bool fresh, const float *sw, int k_steps, uint32_t lane_base, int lane, uint32_t &it,
                                               float (*scales)[32], __nv_bfloat16 *out, long long row_stride, int rows_left) {
    volatile int *abort_flag = &sh.abort;
    __syncwarp();
    uint64_t acc[kCols / 2]; // fp32 pairs
#pragma unroll
    for (int i = 0; i < kCols / 2; ++i) acc[i] = 0;
    const float4 none = make_float4(0.f, 0.f, 0.f, 0.f);
    float4 next_a = valid ? ldScales4(sa_row, 0, k_steps, fresh) : none, next_w = ldScales4(sw, 0, k_steps, false);
    for (int ks0 = 0; ks0 < k_steps; ks0 += 4) {
        // Multiplied now, four steps after the loads; the next four are fetched behind this.
        const float s4[4] = {next_a.x * next_w.x, next_a.y * next_w.y, next_a.z * next_w.z, next_a.w * next_w.w};
        if (ks0 + 4 < k_steps) {
            next_a = valid ? ldScales4(sa_row, ks0 + 4, k_steps, fresh) : none;
            next_w = ldScales4(sw, ks0 + 4, k_steps, false);
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int ks = ks0 + j;
            if (ks >= k_steps) break;
            const int buf = it % kAccBufs;
            const float s = s4[j];
            scales[j & 1][lane] = s; // (the step before may still be read: from the other row)
            __syncwarp();
            if (!mbarWait(&sh.tmemFull[buf], (it / kAccBufs) & 1, abort_flag)) return false;
            tcFenceAfter();
            float v[kCols];
            if constexpr (kCols == 32) tmemLoad32(lane_base + buf * BN, v);
            else tmemLoad16(lane_base + buf * BN, v);
            tmemLoadWait(v);
            tcFenceBefore();
            __syncwarp();
            if (lane == 0) mbarArrive(&sh.tmemEmpty[buf]);
#pragma unroll
            for (int i = 0; i < kCols / 4; ++i) {
                const float4 f = reinterpret_cast<const float4 *>(scales[j & 1])[i];
                asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc[2 * i]) : "l"(pack2(v[4 * i], v[4 * i + 1])), "l"(pack2(f.x, f.y)));
                asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc[2 * i + 1]) : "l"(pack2(v[4 * i + 2], v[4 * i + 3])), "l"(pack2(f.z, f.w)));
            }
            ++it;
        }
    }
    float v[32];
#pragma unroll
    for (int i = 0; i < 16; ++i) {
        if (i < kCols / 2) asm("mov.b64 {%0, %1}, %2;" : "=f"(v[2 * i]), "=f"(v[2 * i + 1]) : "l"(acc[i < kCols / 2 ? i : 0]));
        else v[2 * i] = v[2 * i + 1] = 0.f;
    }
    storeCols32(v, out, row_stride, min(rows_left, kCols), lane);
    return true;
}

struct Tile {
    int g, mt, nt;
};

template<bool kSwapped> __device__ __forceinline__ bool tileAt(const Shared &sh, int groups, int n_tiles, int t, Tile &out) {
    if (t >= sh.tilePrefix[groups]) return false;
    int lo = 0, hi = groups; // tilePrefix[lo] <= t < tilePrefix[hi]
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (sh.tilePrefix[mid] <= t) lo = mid; else hi = mid;
    }
    const int local = t - sh.tilePrefix[lo];
    out.g = lo;
    const int m_tiles = kSwapped ? rowTiles(sh.rowCount[lo]) : 0;
    out.nt = kSwapped ? local / m_tiles : local % n_tiles; // swapped: the row tiles of one W tile side by side
    out.mt = kSwapped ? local - out.nt * m_tiles : local / n_tiles;
    return true;
}

// kSwapped: in a tile of at most 64 rows W is the MMA's M side (128 rows of it), 32 or 64 rows of A are its N side and the accumulator
// is transposed; tiles that share W are neighbours.  With A on the M side every MMA and promotion works on 128 rows however few an
// expert has, and under a steady load the power that takes lowers the clock.  Bound by HBM (W is read once: 537 MB in 90 us, 6.0 TB/s,
// with 4 rows per expert) and, from 32 rows on, by the shared memory that TMA, the MMAs' operands and the scales share.  Tiles of more
// rows keep A on the M side: on the N side they take two tiles, and the same W twice (32 experts of 72 rows 219 us, as now 133), or
// 64 columns per promotion warp with their scales in shared memory (180).
// Measured on one B200, 32 experts, N = K = 4096, back to back, us, A on the M side everywhere / this form: 4 rows each 112 / 90, 16 rows
// 117 / 95, 32 rows 119 / 103, 64 rows 125 / 120, 128 rows 136 / 139; every other expert 70 rows and none between 72 / 73.
template<bool kSwapped>
__global__ void __launch_bounds__(kThreads, 1)
groupedGemmKernel(const __grid_constant__ CUtensorMap mapA, const __grid_constant__ CUtensorMap mapA32, const __grid_constant__ CUtensorMap mapA64,
                  const __grid_constant__ CUtensorMap mapW, const NixlGroupedGemmParams p) {
    extern __shared__ __align__(1024) unsigned char dyn[];
    unsigned char *tiles = reinterpret_cast<unsigned char *>((reinterpret_cast<uintptr_t>(dyn) + 1023) & ~uintptr_t(1023));
    Shared &sh = *reinterpret_cast<Shared *>(tiles + kRingBytes + (kSwapped ? 0 : kTailBytes));
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int n_tiles = p.N / BN, k_steps = p.K / BK;

    if (threadIdx.x == 0) {
        for (int s = 0; s < kMaxStages; ++s) {
            mbarInit(&sh.full[s], 2); // producer (with the byte count) + slot watcher
            mbarInit(&sh.empty[s], 1);
        }
        for (int b = 0; b < kAccBufs; ++b) {
            mbarInit(&sh.tmemFull[b], 1);
            mbarInit(&sh.tmemEmpty[b], 8); // one arrival per promotion warp
        }
        sh.abort = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    nixl_pdl::waitForPreviousKernel(); // (before TMEM is taken: the kernel in front may be about to)
    if (warp == 2) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smemU32(&sh.tmemBase)), "r"(kTmemCols));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    // Tile table: group g owns ceil(count/BM) x n_tiles tiles.
    if (p.counts_flag && threadIdx.x == 0) {
        int run = 0, most = 0;
        // Overlapped with the dispatch: wait for everybody's counts, then derive the rows.
        for (int r = 0; r < p.ranks; ++r) {
            uint64_t t0 = 0;
            unsigned spins = 0;
            while (ldAcquireSys(p.counts_flag + r) < p.epoch) {
                if ((++spins & 63u) == 0) {
                    const uint64_t now = nowNs();
                    if (t0 == 0) t0 = now;
                    else if (now - t0 > p.timeout_ns) {
                        atomicOr(p.status, GEMM_ERR_ARRIVAL);
                        break;
                    }
                }
            }
        }
        int next = 0;
        for (int g = 0; g < p.groups; ++g) {
            int c = 0;
            for (int r = 0; r < p.ranks; ++r) c += p.counts[static_cast<long long>(r) * p.experts_total + p.expert_base + g];
            sh.tilePrefix[g] = run;
            sh.rowStart[g] = p.rows_per_expert > 0 ? g * p.rows_per_expert : next;
            sh.rowCount[g] = c;
            most = max(most, c);
            next += c;
            run += rowTiles(c) * n_tiles;
        }
        sh.tilePrefix[p.groups] = run;
        sh.aRows = aBoxRows(most);
    }
    if (warp == 1 && !p.counts_flag) {
        int most;
        nixl_gemm::buildTileTable(p, n_tiles, rowTiles, sh.tilePrefix, sh.rowStart, sh.rowCount, most);
        if (lane == 0) sh.aRows = aBoxRows(most);
    }
    tcFenceBefore();
    __syncthreads();
    tcFenceAfter();
    // With TMEM in hand: a kernel that moved in before could take it and then wait for this one.  (Not beside a dispatch.)
    if (!p.counts_flag && !p.disp_flag) nixl_pdl::allowNextKernel();
    const uint32_t tmem = sh.tmemBase;
    volatile int *abort_flag = &sh.abort;
    // A stage holds the W tiles and as many A rows as the fullest expert has: with few rows per expert (a decode step) the kernel
    // is bound by the W bytes it keeps in flight, and the room that 128 A rows would take goes to more stages.  It is two steps long
    // so that W comes in boxes of 256 bytes x 128 rows: alone, HBM delivers 6.5 TB/s of those and 6.0 (K = 4096) or 5.3 (K = 7168) of
    // boxes of 128 bytes.
    const uint32_t a_bytes = static_cast<uint32_t>(sh.aRows * BK); // of a step
    const uint32_t stage_bytes = kStageSteps * (kTileBytes + a_bytes);
    const uint32_t stages = min(static_cast<uint32_t>(kMaxStages), kRingBytes / stage_bytes);

    if (warp == 0 && lane == 0) {
        // ---------------------------------------------------------------- TMA producer
        uint32_t s = 0, empty_par = 1; // ring position
        Tile t;
        for (int ti = blockIdx.x; tileAt<kSwapped>(sh, p.groups, n_tiles, ti, t); ti += gridDim.x) {
            const int row0 = sh.rowStart[t.g] + t.mt * BM;
            if (p.disp_flag) {
                waitArrivals(p, t.g, t.mt * BM, min(t.mt * BM + BM, sh.rowCount[t.g]));
                asm volatile("fence.proxy.async;" ::: "memory"); // peers' generic-proxy stores before our async-proxy reads
            }
            const int box = aBoxRows(sh.rowCount[t.g] - t.mt * BM);
            const CUtensorMap *map = box == 32 ? &mapA32 : box == 64 ? &mapA64 : &mapA;
            for (int ks = 0; ks < k_steps; ks += kStageSteps) {
                const bool two = ks + 1 < k_steps;
                if (!mbarWait(&sh.empty[s], empty_par, abort_flag)) goto producer_done;
                mbarExpectTx(&sh.full[s], static_cast<uint32_t>(kStageSteps * kTileBytes + (two ? 2 : 1) * box * BK)); // (W past the end of K arrives as zeros)
                unsigned char *st = tiles + s * stage_bytes;
                tmaLoad3d(st, &mapW, 0, t.g * p.N + t.nt * BN, ks, &sh.full[s]);
                tmaLoad2d(st + kStageSteps * kTileBytes, map, ks * BK, row0, &sh.full[s]);
                if (two) tmaLoad2d(st + kStageSteps * kTileBytes + a_bytes, map, (ks + 1) * BK, row0, &sh.full[s]);
                if (++s == stages) {
                    s = 0;
                    empty_par ^= 1u;
                }
            }
        }
    producer_done:;
    } else if (warp == 1 && lane == 0) {
        // ---------------------------------------------------------------- MMA issuer
        // One barrier per stage: full[s] completes when its bytes have landed (producer) and the
        // TMEM accumulators of its steps are free again (slot watcher), so this thread polls once per
        // eight MMAs, and that poll is started behind the previous stage's MMAs.
        int my_tiles = 0;
        {
            const int total = sh.tilePrefix[p.groups];
            if (static_cast<int>(blockIdx.x) < total) my_tiles = (total - static_cast<int>(blockIdx.x) + static_cast<int>(gridDim.x) - 1) / static_cast<int>(gridDim.x);
        }
        uint32_t s = 0, full_par = 0, buf = 0, ready = 0;
        const uint32_t full_bar0 = smemU32(&sh.full[0]), empty_bar0 = smemU32(&sh.empty[0]), tfull_bar0 = smemU32(&sh.tmemFull[0]);
        const uint64_t desc0 = smemDesc(smemU32(tiles));
        for (int tile = 0; tile < my_tiles; ++tile) {
            uint32_t idesc = instrDesc(BN);
            bool turned = false;
            if constexpr (kSwapped) {
                Tile t;
                tileAt<true>(sh, p.groups, n_tiles, static_cast<int>(blockIdx.x) + tile * static_cast<int>(gridDim.x), t);
                const int rows = sh.rowCount[t.g] - t.mt * BM;
                turned = rows <= kTurned;
                if (turned) idesc = instrDesc(aBoxRows(rows));
            }
            for (int ks = 0; ks < k_steps; ks += kStageSteps) {
                if (!ready && !mbarWait(&sh.full[s], full_par, abort_flag)) goto mma_done;
                tcFenceAfter();
                uint32_t ns = s + 1, nfull_par = full_par;
                if (ns == stages) {
                    ns = 0;
                    nfull_par ^= 1u;
                }
                // Advancing 32 bytes along K inside the swizzle atom = +2 in the 16-byte address field (done in issueStep).
                uint64_t dw = desc0 + static_cast<uint64_t>((s * stage_bytes) >> 4);
                uint64_t da = dw + static_cast<uint64_t>((kStageSteps * kTileBytes) >> 4);
                if (ks + 1 < k_steps) {
                    issueFirstStep(tmem + buf * BN, turned ? dw : da, turned ? da : dw, idesc, tfull_bar0 + buf * 8u);
                    buf = (buf + 1) & (kAccBufs - 1);
                    dw += kTileBytes >> 4;
                    da += a_bytes >> 4;
                }
                issueStep(tmem + buf * BN, turned ? dw : da, turned ? da : dw, idesc, tfull_bar0 + buf * 8u, empty_bar0 + s * 8u, full_bar0 + ns * 8u, nfull_par, ready);
                buf = (buf + 1) & (kAccBufs - 1);
                s = ns;
                full_par = nfull_par;
            }
        }
    mma_done:;
    } else if (warp == 3 && lane == 0) {
        // ---------------------------------------------------------------- slot watcher
        // Adds its arrival to a stage's full[] barrier once the promotion warps have handed back the
        // TMEM accumulators that its steps will write.
        int my_tiles = 0;
        {
            const int total = sh.tilePrefix[p.groups];
            if (static_cast<int>(blockIdx.x) < total) my_tiles = (total - static_cast<int>(blockIdx.x) + static_cast<int>(gridDim.x) - 1) / static_cast<int>(gridDim.x);
        }
        uint32_t s = 0, f_par = 1, buf = 0, e_par = 1;
        bool alive = true;
        for (int tile = 0; tile < my_tiles && alive; ++tile) {
            for (int ks = 0; ks < k_steps && alive; ++ks) {
                alive = mbarWait(&sh.tmemEmpty[buf], e_par, abort_flag);
                buf = (buf + 1) & (kAccBufs - 1);
                if (buf == 0) e_par ^= 1u;
                if (!alive || ((ks & 1) == 0 && ks + 1 < k_steps)) continue; // the stage's second step first
                // The ring may have fewer stages than there are accumulators (K = 128: a step per stage), so that these can be
                // free before the stage's last use has begun: its phase comes first, or it would complete without its bytes.
                alive = mbarWait(&sh.full[s], f_par, abort_flag);
                if (alive) mbarArrive(&sh.full[s]);
                if (++s == stages) {
                    s = 0;
                    f_par ^= 1u;
                }
            }
        }
    } else if (warp >= 4) {
        // ---------------------------------------------------------------- promotion + epilogue
        const int q = warp & 3;            // TMEM lane quarter this warp may touch (fixed by warp id % 4)
        const int half = (warp - 4) >> 2;  // which 64 of the tile's 128 columns this warp promotes
        constexpr int HN = BN / 2;
        const int row_in_tile = q * 32 + lane;
        uint32_t it = 0;
        Tile t;
        const float *scale_a = p.scale_a;
        for (int ti = blockIdx.x; tileAt<kSwapped>(sh, p.groups, n_tiles, ti, t); ti += gridDim.x) {
            const int tile_rows = sh.rowCount[t.g] - t.mt * BM;
            const bool turned = kSwapped && tile_rows <= kTurned;
            const int cols = aBoxRows(tile_rows) / 2; // rows of A that a warp promotes when the operands are swapped
            const int first = t.mt * BM + (turned ? half * cols : q * 32);
            if (first >= sh.rowCount[t.g]) { // this warp's rows are padding: it only hands accumulators back
                bool alive = true;
                for (int ks = 0; ks < k_steps && alive; ++ks, ++it) {
                    alive = mbarWait(&sh.tmemFull[it % kAccBufs], (it / kAccBufs) & 1, abort_flag);
                    if (alive && lane == 0) mbarArrive(&sh.tmemEmpty[it % kAccBufs]);
                }
                if (!alive) break;
                continue;
            }
            const bool fresh = p.disp_flag != nullptr; // the scales travel with the rows
            if (fresh) waitArrivals(p, t.g, first, min(first + 32, sh.rowCount[t.g]));
            if (turned) {
                const int row = first + lane % cols; // whose scales this lane holds
                const float *sa_row = scale_a + (static_cast<long long>(sh.rowStart[t.g]) + row) * k_steps;
                const float *sw = p.scale_w + (static_cast<long long>(t.g) * n_tiles + t.nt) * k_steps;
                const bool valid = row < sh.rowCount[t.g];
                const int rows_left = sh.rowCount[t.g] - first;
                const uint32_t lane_base = tmem + (static_cast<uint32_t>(q * 32) << 16) + half * cols;
                __nv_bfloat16 *out = static_cast<__nv_bfloat16 *>(p.d) + (static_cast<long long>(sh.rowStart[t.g]) + first) * p.N + t.nt * BN + q * 32;
                if (!(cols == 32 ? promoteSwapped<32>(sh, sa_row, valid, fresh, sw, k_steps, lane_base, lane, it, sh.scales[warp - 4], out, p.N, rows_left)
                                 : promoteSwapped<16>(sh, sa_row, valid, fresh, sw, k_steps, lane_base, lane, it, sh.scales[warp - 4], out, p.N, rows_left)))
                    break;
                continue;
            }
            const int local_row = t.mt * BM + row_in_tile;
            const bool valid = local_row < sh.rowCount[t.g];
            const long long grow = static_cast<long long>(sh.rowStart[t.g]) + local_row;
            const float *sa_row = scale_a + grow * k_steps;
            const float *sw = p.scale_w + (static_cast<long long>(t.g) * n_tiles + t.nt) * k_steps;
            uint64_t acc[2][16]; // fp32 pairs
#pragma unroll
            for (int i = 0; i < 16; ++i) acc[0][i] = acc[1][i] = 0;
            bool ok = true;
            // The scales of a step are needed by every FMA of that step, so their loads must not sit on
            // the critical path: they are fetched four steps at a time, four steps ahead, and multiplied when they are there.
            const float4 none = make_float4(0.f, 0.f, 0.f, 0.f);
            float4 next_a = valid ? ldScales4(sa_row, 0, k_steps, fresh) : none, next_w = ldScales4(sw, 0, k_steps, false);
            for (int ks0 = 0; ks0 < k_steps && ok; ks0 += 4) {
                const float s4[4] = {next_a.x * next_w.x, next_a.y * next_w.y, next_a.z * next_w.z, next_a.w * next_w.w};
                if (ks0 + 4 < k_steps) {
                    next_a = valid ? ldScales4(sa_row, ks0 + 4, k_steps, fresh) : none;
                    next_w = ldScales4(sw, ks0 + 4, k_steps, false);
                }
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const int ks = ks0 + j;
                    if (ks >= k_steps) break;
                    const int buf = it % kAccBufs;
                    const float s = s4[j];
                    if (!mbarWait(&sh.tmemFull[buf], (it / kAccBufs) & 1, abort_flag)) {
                        ok = false;
                        break;
                    }
                    tcFenceAfter();
                    const uint32_t base = tmem + (static_cast<uint32_t>(q * 32) << 16) + buf * BN + half * HN;
                    // Two register buffers: the second load is in flight while the first is scaled and added.
                    float v0[32], v1[32];
                    tmemLoad32(base, v0);
                    tmemLoad32(base + 32, v1);
                    tmemLoadWait(v0);
                    tmemLoadWait(v1);
                    // This warp's part of the accumulator has been read: hand it back before the FMAs.
                    tcFenceBefore();
                    __syncwarp();
                    if (lane == 0) mbarArrive(&sh.tmemEmpty[buf]);
                    fmaScale32(acc[0], v0, pack2(s, s));
                    fmaScale32(acc[1], v1, pack2(s, s));
                    ++it;
                }
            }
            if (!ok) break;
            {
                // Coalesced stores (see storeRows64): this thread's 64 columns of its row.
                const int first_row = t.mt * BM + q * 32 + (lane & ~7);
                const long long first_grow = static_cast<long long>(sh.rowStart[t.g]) + first_row;
                const int rows_left = sh.rowCount[t.g] - first_row;
                __nv_bfloat16 *out = static_cast<__nv_bfloat16 *>(p.d) + first_grow * p.N + t.nt * BN + half * HN + (lane & 7) * 8;
                float lo[32], hi[32];
                unpack32(acc[0], lo);
                unpack32(acc[1], hi);
                storeRows64(lo, hi, out, p.N, rows_left, lane);
            }
        }
    }

    tcFenceBefore();
    __syncthreads();
    if (threadIdx.x == 0 && sh.abort) atomicOr(p.status, GEMM_ERR_TIMEOUT);
    if (warp == 2) {
        tcFenceAfter();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols));
    }
}

// ------------------------------------------------------------------ host side

using EncodeFn = CUresult (*)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *, const cuuint64_t *,
                              const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion,
                              CUtensorMapFloatOOBfill);

EncodeFn encoder() {
    static EncodeFn fn = [] {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess || q != cudaDriverEntryPointSuccess)
            p = nullptr;
        return reinterpret_cast<EncodeFn>(p);
    }();
    return fn;
}

} // namespace

bool nixl_gemm::makeTileMap(CUtensorMap *map, const void *base, uint64_t rows, uint64_t k, uint32_t box_rows) {
    EncodeFn fn = encoder();
    if (!fn) return false;
    const cuuint64_t dims[2] = {k, rows};
    const cuuint64_t strides[1] = {k};
    const cuuint32_t box[2] = {BK, box_rows};
    const cuuint32_t elem[2] = {1, 1};
    return fn(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void *>(base), dims, strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE,
              CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

bool nixl_gemm::makePairMap(CUtensorMap *map, const void *base, uint64_t rows, uint64_t k) {
    EncodeFn fn = encoder();
    if (!fn) return false;
    const cuuint64_t dims[3] = {BK, rows, k / BK};
    const cuuint64_t strides[2] = {k, BK};
    const cuuint32_t box[3] = {BK, BN, 2};
    const cuuint32_t elem[3] = {1, 1, 1};
    return fn(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, const_cast<void *>(base), dims, strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE,
              CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// Tile shape: CTA pairs with 256 x 256 tiles when the experts have more rows than one 128-row tile on average and the tiles are
// enough for the 74 pairs; single CTAs with 128 x 128 tiles otherwise (a decode step, where most tiles hold a handful of rows,
// and small products, which need every SM).  The rows are those the caller expects: a's own rows are the capacity of
// the buffer after a dispatch.  Measured back to back, single / pair, us: 32 experts, N = K = 4096: 128 rows each 116 / 122, 200
// rows 210 / 162, 512 rows 477 / 310; 16 experts, 512 x 2048: 256 rows (32 pair tiles) 14.8 / 18.7, 400 rows (50) 22.8 / 19.0;
// 1 expert, 4096 x 7168, 512 rows (32) 27.5 / 35.1.  With the weights out of L2 and room for 160 rows each, 32 experts, N = K =
// 4096: 4 rows each 113 / 125, 32 rows 116 / 123, 64 rows 115 / 125, 128 rows 119 / 125, 160 rows 197 / 152; 2048 x 7168: 32 rows
// 111 / 121, 128 rows 117 / 123, 160 rows 166 / 149.  (The single CTAs' figures are from before their present form, which is faster the
// fewer the rows: 4 rows 93, 32 rows 110, 48 rows and more within 2 percent of those above.  The line stays where it was.)
static long long expectedRows(const NixlGroupedGemmParams &p) { return p.expected_rows > 0 && p.expected_rows < p.a_rows ? p.expected_rows : p.a_rows; }

extern "C" int nixl_grouped_gemm_fp8_mode(const NixlGroupedGemmParams *params) {
    const NixlGroupedGemmParams &p = *params;
    if (const int asked = p.tile_mode & 0xff) return asked;
    const long long rows = expectedRows(p);
    return p.rows_per_expert == 0 && !p.counts_flag && p.N % 256 == 0 && rows > 128LL * p.groups && rows * p.N >= 40LL * 256 * 256 ? 2 : 1;
}

// Single CTAs with swapped operands (see groupedGemmKernel) up to 40 expected rows per expert: us, A on the M side everywhere / swapped,
// for 32 experts, N = K = 4096: 32 rows each 119 / 103, 48 rows 124 / 118, 64 rows 125 / 120, 72 rows 130 / 133.  Between 40 and 64 rows
// uneven routing puts more and more experts above 64, where this form gains nothing.
static bool swappedTiles(const NixlGroupedGemmParams &p) { return expectedRows(p) <= 40LL * p.groups; }

extern "C" int nixl_grouped_gemm_fp8_launch(const NixlGroupedGemmParams *params, void *stream) {
    if (!params || !params->a || !params->w || !params->d || !params->scale_a || !params->scale_w || !params->status)
        return cudaErrorInvalidValue;
    if (!params->counts_flag && (!params->row_start || !params->row_count)) return cudaErrorInvalidValue;
    const NixlGroupedGemmParams &p = *params;
    if (p.groups <= 0 || p.groups > kMaxGroups || p.N <= 0 || p.N % BN || p.K <= 0 || p.K % BK || p.a_rows <= 0)
        return cudaErrorInvalidValue;
    if ((reinterpret_cast<uintptr_t>(p.a) | reinterpret_cast<uintptr_t>(p.w) | reinterpret_cast<uintptr_t>(p.d)) & 15) return cudaErrorInvalidValue;
    if ((p.disp_flag || p.counts_flag) && (!p.counts || p.ranks <= 0)) return cudaErrorInvalidValue;
    const uint64_t a_rows = static_cast<uint64_t>(p.a_rows), k_bytes = static_cast<uint64_t>(p.K);
    CUtensorMap mapW, mapA, mapA32, mapA64; // A in boxes of 128, 32 and 64 rows
    const uint64_t w_rows = static_cast<uint64_t>(p.groups) * p.N;
    const int mode = nixl_grouped_gemm_fp8_mode(&p);
    if (!(mode == 2 || mode == 3 ? nixl_gemm::makeTileMap(&mapW, p.w, w_rows, k_bytes) : nixl_gemm::makePairMap(&mapW, p.w, w_rows, k_bytes)) ||
        !nixl_gemm::makeTileMap(&mapA64, p.a, a_rows, k_bytes, 64)) {
        std::fprintf(stderr, "nixl_grouped_gemm_fp8_launch: cuTensorMapEncodeTiled failed\n");
        return cudaErrorInvalidValue;
    }
    if (mode == 3) {
        if (p.N % 256 || p.K % 512 || p.counts_flag || p.disp_flag) return cudaErrorInvalidValue;
        if ((reinterpret_cast<uintptr_t>(p.scale_a) | reinterpret_cast<uintptr_t>(p.scale_w)) & 3) return cudaErrorInvalidValue;
        CUtensorMap mapW2;
        if (!nixl_gemm::makeTileMap(&mapA, p.a, a_rows, k_bytes) || !nixl_gemm::makeTileMap(&mapA32, p.a, a_rows, k_bytes, 32) ||
            !nixl_gemm::makePairMap(&mapW2, p.w, w_rows, k_bytes))
            return cudaErrorInvalidValue;
        return nixl_gemm::launchMxPairKernel(mapA, mapA32, mapA64, mapW, mapW2, p, static_cast<cudaStream_t>(stream));
    }
    if (mode == 2) {
        if (p.N % 256) return cudaErrorInvalidValue;
        if (!nixl_gemm::makeTileMap(&mapA, p.a, a_rows, k_bytes)) return cudaErrorInvalidValue;
        return nixl_gemm::launchPairKernel(mapA, mapA64, mapW, p, static_cast<cudaStream_t>(stream));
    }
    if (!nixl_gemm::makeTileMap(&mapA, p.a, a_rows, k_bytes) || !nixl_gemm::makeTileMap(&mapA32, p.a, a_rows, k_bytes, 32)) return cudaErrorInvalidValue;
    const bool swapped = swappedTiles(p);
    const auto kernel = swapped ? groupedGemmKernel<true> : groupedGemmKernel<false>;
    const size_t smem = size_t(kRingBytes) + (swapped ? 0 : kTailBytes) + sizeof(Shared) + 1024;
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    {
        // The shared-memory limit is a per-device function attribute.
        static bool attr_done[2][64] = {};
        if (dev >= 0 && dev < 64 && !attr_done[swapped][dev]) {
            cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
            if (e != cudaSuccess) return e;
            attr_done[swapped][dev] = true;
        }
    }
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    int grid = p.grid > 0 ? p.grid : sms;
    // Upper bound of tiles (row counts live on the device): never launch more CTAs than that.
    const long long max_tiles = (static_cast<long long>(p.a_rows + BM - 1) / BM + p.groups) * (p.N / BN);
    if (grid > max_tiles) grid = static_cast<int>(max_tiles);
    if (p.counts_flag || p.disp_flag) { // waits for a dispatch on another stream: not before the stream's own turn
        kernel<<<grid, kThreads, smem, static_cast<cudaStream_t>(stream)>>>(mapA, mapA32, mapA64, mapW, p);
        return cudaGetLastError();
    }
    return nixl_pdl::launch(kernel, grid, kThreads, smem, static_cast<cudaStream_t>(stream), mapA, mapA32, mapA64, mapW, p);
}
