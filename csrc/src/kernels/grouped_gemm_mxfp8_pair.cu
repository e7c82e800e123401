// Grouped fp8 expert GEMM with power-of-two (UE8M0) block scales applied by the tensor core:
// tcgen05.mma.kind::mxf8f6f4.block_scale on CTA pairs, 256 x 256 output tiles.
//
//   D[rows of expert g, :] = (A * 2^(sa-127)) x (W[g] * 2^(sw-127))^T           (bf16 out)
//   A: e4m3 [rows][K], one biased exponent byte per row per 128 channels (what EP dispatch delivers
//      with use_ue8m0: uint8 [rows][K/128], i.e. four consecutive steps per 32-bit word)
//   W: e4m3 [G][N][K], one exponent byte per 128 x 128 block: uint8 [G][N/128][K/128]
//
// With fp32 scales the partial sums of every 128-channel step have to leave TMEM to be scaled
// (grouped_gemm_fp8_pair.cu), and that promotion, not the tensor pipe, bounds the kernel.  Here the
// scale factors ride along with the MMA: a whole K loop accumulates in TMEM and the epilogue runs
// once per tile.
//
// The roles of the operands are swapped: W is the MMA's M side (256 weight rows per pair, 128 per CTA) and the tokens
// are its N side.  N may be any multiple of 32, so an expert's rows are split into equal tiles of at most 256 tokens,
// rounded up to 32, and almost nothing is computed, loaded or kept in TMEM for padding; with the tokens on the M side every
// expert's last tile cost 256 rows.  The accumulator is transposed (a lane is a column of D, a TMEM column a token), which
// the epilogue undoes with shuffles between neighbouring lanes (storeCols32).
//
// Scale factors reach the tensor core through TMEM.  For four steps at a time ("chunk") the
// epilogue warps, idle during the main loop, build in shared memory the 512-byte layouts the
// hardware wants (byte (r % 32) * 16 + (r / 32) * 4 + step for row r: for the tokens one 32-bit word per row
// straight from the scale tensor, for W the block's word repeated for all 128 rows), the issuing
// thread copies them to TMEM with tcgen05.cp (32x128b.warpx4) and selects the step's byte with the
// scale-factor-id fields of the instruction descriptor.  The copies run in the MMAs' pipe, and each run of them is a
// bubble there; up to eight chunks (4096 channels) are therefore copied at once.  Both the shared-memory buffers and
// the TMEM scale columns are double-buffered by such groups.
//
//   warp 0      TMA producer (both CTAs; bytes counted on the even CTA's barrier)
//   warps 1, 3  MMA issuers (even CTA): tcgen05.cp of scale groups, four M256 K32 MMAs per step
//   warp 2      TMEM allocator (512 columns: 256 accumulator, 192 scale factors)
//   warps 4-11  scale staging during the main loop, then the epilogue (TMEM -> bf16 -> global)
//
// Bound by power: the SM clock is 1.55 GHz at the first launch and 1.25 to 1.4 GHz after half a second; a full step takes
// 697 cycles of which the MMAs need 512.  What is left is mostly the traffic into shared memory (64 of 128 bytes per cycle
// at full rate, beside the operands' reads).  The cap by itself would allow more: a library's plain fp8 product (8192 cubed, no block
// scales, the same random inputs) settles at 2.65 PFLOP/s and 1.34 GHz (3.08 as a burst), this kernel, with experts of whole
// tiles, at 1.97 (2048 x 7168) to 2.10 (4096 x 4096) and 1.06 to 1.24 GHz (2.36 to 2.43): it spends more energy per operation,
// where is not known.  Measured on one B200 back to back for half a second, before (tokens on the
// M side, eight N = 128 MMAs per step, scale copies every 512 channels) / now: 31 experts that share 16384 rows unevenly,
// 2048 x 7168: 335 / 277 us (1.74 PFLOP/s); 32 experts, 32768 rows, 4096 x 4096: 659 / 562 us (1.96 PFLOP/s); one
// expert, 8192 rows, 4096 x 7168: 239 / 200 us (2.41 PFLOP/s); 32 experts, 1024 rows, 2048 x 7168: 130 / 97 us.
//
// TMA loads read this GPU's memory only and carry no cluster multicast.  Every wait is bounded.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include "kernels/grouped_gemm_internal.h"
#include "kernels/programmatic_launch.cuh"
#include "kernels/tcgen05_ptx.cuh"

namespace {

using namespace nixl_tc;
using nixl_gemm::GEMM_ERR_TIMEOUT;
using nixl_gemm::kMaxGroups;

constexpr int BW = 128;        // W rows per CTA (256 per pair): the MMA's M side
constexpr int BT = 256;        // tokens per tile at most: its N side, half of them from either CTA
constexpr int BK = 128;
constexpr int kMaxStages = 6;
constexpr int kThreads = 384;
constexpr int kWTileBytes = BW * BK;
constexpr uint32_t kOneStepStage = kWTileBytes + BT / 2 * BK; // 32 KiB
constexpr int kRingBytes = kMaxStages * kOneStepStage; // 192 KiB per CTA
constexpr int kChunkSteps = 4;                 // steps whose scale bytes share one 32-bit word
constexpr int kGroupChunks = 8;                // chunks copied to TMEM in one go
constexpr int kSfAtomBytes = 512;              // 128 rows x 4 steps
constexpr int kSfChunkBytes = 3 * kSfAtomBytes;  // tokens 0 .. 127, tokens 128 .. 255, W
constexpr int kSfBufBytes = kGroupChunks * kSfChunkBytes;
constexpr int kTmemCols = 512;
constexpr int kAccCols = BT;                   // accumulator: columns [0, 256)
constexpr int kSfTmemChunk = 12;               // scale columns of a chunk: tokens +0 .. +7, W +8 .. +11
constexpr int kSfTmemStride = kGroupChunks * kSfTmemChunk; // of a group; group g uses [256 + 96 (g % 2), ...)
constexpr int kPromoWarps = 8;
static_assert(kAccCols + 2 * kSfTmemStride <= kTmemCols, "accumulator and scale columns share TMEM");

struct Shared {
    uint64_t full[kMaxStages];   // even CTA: both CTAs' operand bytes of a stage have landed
    uint64_t empty[kMaxStages];  // per CTA: the MMAs that read the stage are done
    uint64_t sfFull[2];          // even CTA: both CTAs have staged the group's scale layouts (16 warp arrivals)
    uint64_t sfEmpty[2];         // per CTA: the group's buffer has been copied to TMEM
    uint64_t tmemFull;           // per CTA: a tile's accumulator is complete
    uint64_t tmemEmpty;          // even CTA: all 16 epilogue warps have read the accumulator
    uint32_t tmemBase;
    int abort;
    uint32_t chunksIssued;       // two issuing threads take turns chunk by chunk: the next chunk whose MMAs may enter the pipe
    int tilePrefix[kMaxGroups + 1];
    int rowStart[kMaxGroups];
    int rowCount[kMaxGroups];
    int tileRows[kMaxGroups]; // tokens per tile of the group, a multiple of 32
    int boxRows;                 // tokens of a CTA that a step has room for: 32, 64 or 128
};

__device__ __forceinline__ uint32_t clusterCtaRank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ uint32_t mapToCta(uint32_t smem_addr, uint32_t cta) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(smem_addr), "r"(cta));
    return r;
}
__device__ __forceinline__ void clusterSync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// Relaxed on purpose: a release at cluster scope made the arriving thread wait several hundred
// cycles, once per slot.  What the arrive has to order are this warp's TMEM reads, and those are
// complete (tcgen05.wait::ld returned, the values are in registers) before it is issued.
__device__ __forceinline__ void mbarArriveCluster(uint32_t cluster_addr) {
    asm volatile("mbarrier.arrive.relaxed.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
// Tile load whose completion bytes are counted on a barrier given by its cluster address
// (the even CTA's), as the paired MMA needs both halves before it may start.
__device__ __forceinline__ void tmaLoad2dPair(void *smem_dst, const CUtensorMap *map, int x, int y, uint32_t bar_cluster_addr) {
    asm volatile("cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::"r"(
                     smemU32(smem_dst)),
                 "l"(map), "r"(bar_cluster_addr), "r"(x), "r"(y)
                 : "memory");
}
__device__ __forceinline__ void tmaLoad3dPair(void *smem_dst, const CUtensorMap *map, int x, int y, int z, uint32_t bar_cluster_addr) {
    asm volatile("cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];" ::"r"(
                     smemU32(smem_dst)),
                 "l"(map), "r"(bar_cluster_addr), "r"(x), "r"(y), "r"(z)
                 : "memory");
}
__device__ __forceinline__ void mbarArriveClusterRelease(uint32_t cluster_addr) {
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
__device__ __forceinline__ void tcCommitPair(uint32_t bar_addr) {
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar_addr),
                 "h"(static_cast<uint16_t>(3))
                 : "memory");
}
// Shared-memory descriptor of one 512-byte scale layout: 32 rows of 16 bytes, no swizzle, 8-row
// groups 128 bytes apart.
__device__ __forceinline__ uint64_t sfDesc(uint32_t smem_addr) {
    uint64_t d = 0;
    d |= static_cast<uint64_t>((smem_addr & 0x3FFFFu) >> 4);
    d |= static_cast<uint64_t>(1) << 16;
    d |= static_cast<uint64_t>(128 >> 4) << 32;
    d |= static_cast<uint64_t>(1) << 46;
    return d;
}
// 32 x 128 bit from shared memory into four TMEM columns, replicated to all four lane quarters, in
// both CTAs of the pair (each from its own shared memory).
__device__ __forceinline__ void tmemCpPair(uint32_t tmem_dst, uint64_t desc) {
    asm volatile("tcgen05.cp.cta_group::2.32x128b.warpx4 [%0], %1;" ::"r"(tmem_dst), "l"(desc) : "memory");
}
// D fp32, A and B e4m3 K-major, M = 256 (both CTAs), N = n, scale factors E8M0, scale-factor id `sf` for A and B.
__device__ __forceinline__ uint32_t instrDescMx(uint32_t sf, uint32_t n) {
    return (sf << 4) | ((n >> 3) << 17) | (1u << 23) | (static_cast<uint32_t>((2 * BW) >> 4) << 24) | (sf << 29);
}

// The first of a stage's two steps: its four MMAs.
__device__ __forceinline__ void issueFirstStepMx(uint32_t tmem_d, uint64_t dw, uint64_t dt, uint32_t idesc, uint32_t tsfw, uint32_t tsft, uint32_t accumulate) {
    asm volatile(
        "{\n"
        " .reg .pred pacc, pfirst;\n"
        " setp.ne.b32 pacc, %7, 0;\n"
        " setp.ne.b32 pfirst, %6, 0;\n"
        " tcgen05.mma.cta_group::2.kind::mxf8f6f4.block_scale [%0], %1, %2, %3, [%4], [%5], pfirst;\n"
        " add.u64 %1, %1, 2;\n add.u64 %2, %2, 2;\n"
        " tcgen05.mma.cta_group::2.kind::mxf8f6f4.block_scale [%0], %1, %2, %3, [%4], [%5], pacc;\n"
        " add.u64 %1, %1, 2;\n add.u64 %2, %2, 2;\n"
        " tcgen05.mma.cta_group::2.kind::mxf8f6f4.block_scale [%0], %1, %2, %3, [%4], [%5], pacc;\n"
        " add.u64 %1, %1, 2;\n add.u64 %2, %2, 2;\n"
        " tcgen05.mma.cta_group::2.kind::mxf8f6f4.block_scale [%0], %1, %2, %3, [%4], [%5], pacc;\n"
        "}\n"
        : "+r"(tmem_d), "+l"(dw), "+l"(dt)
        : "r"(idesc), "r"(tsfw), "r"(tsft), "r"(accumulate), "r"(1u)
        : "memory");
}

// One 128-channel step: four block-scaled MMAs and the commit that frees the stage.  The non-blocking
// test of the next step's barrier sits between the MMAs: its latency then runs while the others are
// being issued, and its result is read last.
__device__ __forceinline__ void issueKStepMx(uint32_t tmem_d, uint64_t dw, uint64_t dt, uint32_t idesc, uint32_t tsfw, uint32_t tsft, uint32_t accumulate,
                                             uint32_t bar_stage_empty, uint32_t peek_bar, uint32_t peek_par, uint32_t &ready_next) {
    asm volatile(
        "{\n"
        " .reg .pred pf, pacc, pfirst;\n"
        " setp.ne.b32 pacc, %11, 0;\n"
        " setp.ne.b32 pfirst, %7, 0;\n"
        " tcgen05.mma.cta_group::2.kind::mxf8f6f4.block_scale [%1], %2, %3, %4, [%5], [%6], pfirst;\n"
        " add.u64 %2, %2, 2;\n add.u64 %3, %3, 2;\n"
        " tcgen05.mma.cta_group::2.kind::mxf8f6f4.block_scale [%1], %2, %3, %4, [%5], [%6], pacc;\n"
        " mbarrier.test_wait.parity.shared::cta.b64 pf, [%9], %10;\n"
        " add.u64 %2, %2, 2;\n add.u64 %3, %3, 2;\n"
        " tcgen05.mma.cta_group::2.kind::mxf8f6f4.block_scale [%1], %2, %3, %4, [%5], [%6], pacc;\n"
        " add.u64 %2, %2, 2;\n add.u64 %3, %3, 2;\n"
        " tcgen05.mma.cta_group::2.kind::mxf8f6f4.block_scale [%1], %2, %3, %4, [%5], [%6], pacc;\n"
        " tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%8], %12;\n"
        " selp.u32 %0, 1, 0, pf;\n"
        "}\n"
        : "=r"(ready_next), "+r"(tmem_d), "+l"(dw), "+l"(dt)
        : "r"(idesc), "r"(tsfw), "r"(tsft), "r"(accumulate), "r"(bar_stage_empty), "r"(peek_bar), "r"(peek_par), "r"(1u), "h"(static_cast<uint16_t>(3))
        : "memory");
}

// Rows of the one TMA box that fetches a CTA's half of a tile: an instruction more per step costs more than the rows it would save.
__device__ __forceinline__ int boxRows(int half) { return half <= 32 ? 32 : half <= 64 ? 64 : BT / 2; }

struct Tile {
    int g, mt, nt;
};

__device__ __forceinline__ bool tileAt(const Shared &sh, int groups, int n_tiles, int t, Tile &out) {
    if (t >= sh.tilePrefix[groups]) return false;
    int lo = 0, hi = groups;
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (sh.tilePrefix[mid] <= t) lo = mid; else hi = mid;
    }
    const int local = t - sh.tilePrefix[lo];
    out.g = lo;
    out.mt = local / n_tiles;
    out.nt = local - out.mt * n_tiles;
    return true;
}

// One issuing thread's share of a pair's chunks.  kTwo: stages of two steps (see the kernel).
template<bool kTwo>
__device__ __forceinline__ void issueChunks(Shared &sh, unsigned char *tiles, unsigned char *sf_ring, const NixlGroupedGemmParams &p, int n_tiles, int chunks, int sf_groups, int pair,
                                            int pairs, int my_tiles, uint32_t me, uint32_t tmem, uint32_t stage_bytes, uint32_t stages) {
    constexpr uint32_t kSteps = kTwo ? 2 : 1; // of a stage
    volatile int *abort_flag = &sh.abort;
    const uint32_t full_bar0 = smemU32(&sh.full[0]), empty_bar0 = smemU32(&sh.empty[0]), sfempty_bar0 = smemU32(&sh.sfEmpty[0]);
    const uint64_t desc0 = smemDesc(smemU32(tiles));
    const uint32_t sf_smem0 = smemU32(sf_ring);
    const uint32_t total_chunks = static_cast<uint32_t>(my_tiles) * static_cast<uint32_t>(chunks);
    uint32_t known_tile = 0xffffffffu, n_tokens = 32;
    for (uint32_t cc = me; cc < total_chunks; cc += 2) {
        const uint32_t tile = cc / static_cast<uint32_t>(chunks), c = cc - tile * static_cast<uint32_t>(chunks);
        const uint32_t it0 = cc * (kChunkSteps / kSteps); // the chunk's first use of a stage
        uint32_t s = it0 % stages, full_par = (it0 / stages) & 1u;
        const uint32_t gg = tile * static_cast<uint32_t>(sf_groups) + c / kGroupChunks, b = gg & 1u; // scale group
        if (tile != known_tile) {
            Tile t;
            if (tileAt(sh, p.groups, n_tiles, pair + static_cast<int>(tile) * pairs, t)) n_tokens = static_cast<uint32_t>(sh.tileRows[t.g]);
            known_tile = tile;
        }
        // Everything this chunk depends on, before asking for the turn.
        if (c % kGroupChunks == 0 && !mbarWait(&sh.sfFull[b], (gg >> 1) & 1u, abort_flag)) return;
        if (!mbarWait(&sh.full[s], full_par, abort_flag)) return;
        {
            const long long t0 = clock64();
            while (ldAcquireCta(&sh.chunksIssued) != cc) {
                if (*abort_flag) return;
                if (clock64() - t0 > (1ll << 33)) {
                    *abort_flag = 1;
                    return;
                }
            }
        }
        // Accumulator drained by the previous tile's epilogue.  With the turn in hand, not before: the previous tile is
        // then issued, so its own wait here has passed and the barrier is at most one phase behind, which is all a parity
        // can tell.  (With one chunk per tile a thread would otherwise look before the other one issued the tile between,
        // two phases early, and pass at once.)
        if (c == 0 && !mbarWait(&sh.tmemEmpty, (tile & 1u) ^ 1u, abort_flag)) return;
        tcFenceAfter();
        const uint32_t sf_base = tmem + kAccCols + b * kSfTmemStride;
        if (c % kGroupChunks == 0) {
            const uint32_t here = min(static_cast<uint32_t>(kGroupChunks), static_cast<uint32_t>(chunks) - c);
            for (uint32_t i = 0; i < here; ++i) {
                const uint32_t src = sf_smem0 + b * kSfBufBytes + i * kSfChunkBytes, dst = sf_base + i * kSfTmemChunk;
                tmemCpPair(dst, sfDesc(src));
                if (n_tokens > 128) tmemCpPair(dst + 4, sfDesc(src + kSfAtomBytes));
                tmemCpPair(dst + 8, sfDesc(src + 2 * kSfAtomBytes));
            }
            tcCommitPair(sfempty_bar0 + b * 8u); // the buffer may be refilled once the copies have read it
        }
        const uint32_t sfc = sf_base + (c % kGroupChunks) * kSfTmemChunk;
        uint32_t ready = 1; // the first stage's barrier was waited for above
#pragma unroll
        for (uint32_t sub = 0; sub < kChunkSteps; ++sub) {
            const uint32_t odd = kTwo ? sub & 1u : 0u; // a stage's second step
            if (!odd) {
                if (!ready && !mbarWait(&sh.full[s], full_par, abort_flag)) return;
                tcFenceAfter();
            }
            const uint64_t dw = desc0 + static_cast<uint64_t>((s * stage_bytes + odd * kWTileBytes) >> 4);
            const uint64_t dt = desc0 + static_cast<uint64_t>((s * stage_bytes + kSteps * kWTileBytes + odd * (stage_bytes / kSteps - kWTileBytes)) >> 4);
            const uint32_t accumulate = (c | sub) ? 1u : 0u;
            if (kTwo && !odd) {
                issueFirstStepMx(tmem, dw, dt, instrDescMx(sub, n_tokens), sfc + 8, sfc, accumulate);
                continue;
            }
            uint32_t ns = s + 1, nfull_par = full_par;
            if (ns == stages) {
                ns = 0;
                nfull_par ^= 1u;
            }
            issueKStepMx(tmem, dw, dt, instrDescMx(sub, n_tokens), sfc + 8, sfc, accumulate, empty_bar0 + s * 8u, full_bar0 + ns * 8u, nfull_par, ready);
            s = ns;
            full_par = nfull_par;
        }
        // All of this chunk's MMAs are in the pipe: the other thread's chunk may follow.  It adds to the accumulator
        // these MMAs write and may read the scale columns copied here, and tcgen05 operations of two threads are in
        // order only across a fence on either side of the hand-over (tcFenceAfter: above, with the turn).
        tcFenceBefore();
        stReleaseCta(&sh.chunksIssued, cc + 1);
        if (c + 1 == static_cast<uint32_t>(chunks) || c + 2 == static_cast<uint32_t>(chunks)) {
            // This thread's last chunk of the tile: its share of "accumulator complete" (both shares when
            // the tile has a single chunk and the other thread never touches it).
            tcCommitPair(smemU32(&sh.tmemFull));
            if (chunks == 1) tcCommitPair(smemU32(&sh.tmemFull));
        }
    }
}

__global__ void __launch_bounds__(kThreads, 1)
groupedGemmMxPairKernel(const __grid_constant__ CUtensorMap mapT, const __grid_constant__ CUtensorMap mapT32, const __grid_constant__ CUtensorMap mapT64,
                        const __grid_constant__ CUtensorMap mapW, const __grid_constant__ CUtensorMap mapW2, const NixlGroupedGemmParams p) {
    extern __shared__ __align__(1024) unsigned char dyn[];
    unsigned char *tiles = reinterpret_cast<unsigned char *>((reinterpret_cast<uintptr_t>(dyn) + 1023) & ~uintptr_t(1023));
    unsigned char *sf_ring = tiles + kRingBytes; // two buffers of kGroupChunks chunks' layouts
    Shared &sh = *reinterpret_cast<Shared *>(sf_ring + 2 * kSfBufBytes);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int n_tiles = p.N / (2 * BW), k_steps = p.K / BK;
    const int chunks = k_steps / kChunkSteps; // K is a multiple of 512
    const int sf_groups = (chunks + kGroupChunks - 1) / kGroupChunks; // per tile
    const uint32_t cta = clusterCtaRank();
    const int pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;

    if (threadIdx.x == 0) {
        for (int s = 0; s < kMaxStages; ++s) {
            mbarInit(&sh.full[s], 1);
            mbarInit(&sh.empty[s], 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbarInit(&sh.sfFull[b], 2 * kPromoWarps);
            mbarInit(&sh.sfEmpty[b], 1);
        }
        mbarInit(&sh.tmemFull, 2); // one commit from each issuing thread
        mbarInit(&sh.tmemEmpty, 2 * kPromoWarps);
        sh.abort = 0;
        sh.chunksIssued = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    nixl_pdl::waitForPreviousKernel(); // (before TMEM is taken: the kernel in front may be about to)
    if (warp == 2) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smemU32(&sh.tmemBase)), "r"(kTmemCols));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;");
    }
    if (warp == 1) {
        int most;
        nixl_gemm::buildTileTable(p, n_tiles, [](int rows) { return (rows + BT - 1) / BT; }, sh.tilePrefix, sh.rowStart, sh.rowCount, most);
        int widest = 32;
        for (int g = lane; g < p.groups; g += 32) { // (each lane wrote its groups' counts itself)
            const int c = sh.rowCount[g], tiles_g = (c + BT - 1) / BT; // equal tiles, rounded up to the MMA's granularity
            sh.tileRows[g] = tiles_g > 0 ? ((c + tiles_g - 1) / tiles_g + 31) & ~31 : 32;
            widest = max(widest, sh.tileRows[g]);
        }
        widest = __reduce_max_sync(0xffffffffu, widest);
        if (lane == 0) sh.boxRows = boxRows(widest / 2);
    }
    tcFenceBefore();
    __syncthreads();
    clusterSync();
    tcFenceAfter();
    nixl_pdl::allowNextKernel(); // (with TMEM in hand: a kernel that moved in before could take it and then wait for this one)
    const uint32_t tmem = sh.tmemBase;
    volatile int *abort_flag = &sh.abort;
    // With at most 128 tokens in any tile the kernel is bound by W from HBM: a stage then holds two steps, so that W comes in boxes of
    // 256 bytes x 128 rows, and the room that wider tiles would take goes to more steps in flight (eight instead of six): 32 experts,
    // 1024 rows, 2048 x 7168 100 -> 94 us; 40 experts, 9000 rows, 1024 x 3584 60 -> 55 (2 of them by the launch).  Wider tiles keep
    // stages of one step: with two, 32 experts, 32768 rows, 4096 x 4096 took 558 us instead of 550.
    const bool two = sh.boxRows <= 64;
    const uint32_t stage_steps = two ? 2 : 1;
    const uint32_t t_bytes = static_cast<uint32_t>(sh.boxRows * BK); // of a step
    const uint32_t stage_bytes = stage_steps * (kWTileBytes + t_bytes);
    const uint32_t stages = min(static_cast<uint32_t>(kMaxStages), kRingBytes / stage_bytes);
    int my_tiles = 0;
    {
        const int total = sh.tilePrefix[p.groups];
        if (pair < total) my_tiles = (total - pair + pairs - 1) / pairs;
    }

    if (warp == 0 && lane == 0) {
        // ---------------------------------------------------------------- TMA producer (both CTAs)
        const uint32_t full0 = mapToCta(smemU32(&sh.full[0]), 0);
        uint32_t s = 0, empty_par = 1; // ring position
        Tile t;
        for (int ti = pair; tileAt(sh, p.groups, n_tiles, ti, t); ti += pairs) {
            const int half = sh.tileRows[t.g] / 2; // tokens of this CTA
            const int row0 = sh.rowStart[t.g] + t.mt * (2 * half) + static_cast<int>(cta) * half;
            const int wrow = t.g * p.N + t.nt * (2 * BW) + static_cast<int>(cta) * BW;
            const int box = boxRows(half);
            const CUtensorMap *map = box == 32 ? &mapT32 : box == 64 ? &mapT64 : &mapT;
            const uint32_t bytes = 2 * stage_steps * static_cast<uint32_t>(kWTileBytes + box * BK); // both CTAs' shares
            for (int ks = 0; ks < k_steps; ks += static_cast<int>(stage_steps)) {
                if (!mbarWait(&sh.empty[s], empty_par, abort_flag)) goto producer_done;
                if (cta == 0) mbarExpectTx(&sh.full[s], bytes);
                const uint32_t bar = full0 + s * 8u;
                unsigned char *st = tiles + s * stage_bytes;
                unsigned char *tokens = st + stage_steps * kWTileBytes;
                if (two) {
                    tmaLoad3dPair(st, &mapW2, 0, wrow, ks, bar);
                    tmaLoad2dPair(tokens + t_bytes, map, (ks + 1) * BK, row0, bar);
                } else {
                    tmaLoad2dPair(st, &mapW, ks * BK, wrow, bar);
                }
                tmaLoad2dPair(tokens, map, ks * BK, row0, bar);
                if (++s == stages) {
                    s = 0;
                    empty_par ^= 1u;
                }
            }
        }
    producer_done:;
    } else if ((warp == 1 || warp == 3) && lane == 0 && cta == 0) {
        // ---------------------------------------------------------------- two MMA issuers (even CTA)
        // The tensor pipe idles whenever its issuing thread does anything but issue (an MMA's issue
        // returns about when its predecessor starts).  Two threads therefore alternate chunk by chunk
        // (four steps, 16 MMAs): while one is parked in the issue of its chunk, the other waits for its
        // next chunk's barriers and sits ready.  A turn counter keeps the chunks entering the pipe in
        // order (the first step of a tile overwrites the accumulator, and the scale copies of a group of up to eight
        // chunks, made by the thread that has its first one, must precede the MMAs of both threads that read them);
        // even groups use one set of TMEM scale columns, odd groups the other.
        const uint32_t me = warp == 1 ? 0u : 1u;
        if (two) issueChunks<true>(sh, tiles, sf_ring, p, n_tiles, chunks, sf_groups, pair, pairs, my_tiles, me, tmem, stage_bytes, stages);
        else issueChunks<false>(sh, tiles, sf_ring, p, n_tiles, chunks, sf_groups, pair, pairs, my_tiles, me, tmem, kOneStepStage, kMaxStages);
    } else if (warp >= 4) {
        // ---------------------------------------------------------------- scale staging, then the epilogue
        const int q = warp & 3;
        const int part = (warp - 4) >> 2; // epilogue: which half of the tile's tokens
        const int row = (warp - 4) * 32 + lane; // staging: token of the tile
        const uint32_t sffull0 = mapToCta(smemU32(&sh.sfFull[0]), 0);
        const uint32_t tempty = mapToCta(smemU32(&sh.tmemEmpty), 0);
        const uint32_t lane_base = tmem + (static_cast<uint32_t>(q * 32) << 16);
        const uint32_t *sa32 = reinterpret_cast<const uint32_t *>(p.scale_a);
        const uint32_t *sw32 = reinterpret_cast<const uint32_t *>(p.scale_w);
        const int n_blocks = p.N / 128;
        // Builds the layouts of scale group sg of a tile in buffer gcc % 2 once the issuer has copied that buffer's previous content out.
        auto stage = [&](const Tile &t, int sg, uint32_t gcc) -> bool {
            const uint32_t b = gcc & 1u;
            if (!mbarWait(&sh.sfEmpty[b], ((gcc >> 1) & 1u) ^ 1u, abort_flag)) return false;
            uint32_t *buf = reinterpret_cast<uint32_t *>(sf_ring + b * kSfBufBytes);
            const int c0 = sg * kGroupChunks, here = min(kGroupChunks, chunks - c0);
            const int local = t.mt * sh.tileRows[t.g] + row;
            const bool valid = row < sh.tileRows[t.g] && local < sh.rowCount[t.g];
            const uint32_t *sa = sa32 + (static_cast<long long>(sh.rowStart[t.g]) + (valid ? local : 0)) * chunks + c0;
            const uint32_t *sw = sw32 + (static_cast<long long>(t.g) * n_blocks + t.nt * 2 + static_cast<int>(cta)) * chunks + c0;
#pragma unroll
            for (int i = 0; i < kGroupChunks; ++i) {
                if (i >= here) break;
                uint32_t *layout = buf + i * (kSfChunkBytes / 4);
                // Token r: word (r % 32) * 4 + r / 32 of its 128 tokens' layout (rows beyond the expert get exponent 127 = 1.0).
                layout[part * 128 + lane * 4 + q] = valid ? nixl_gemm::ldExponents(sa + i) : 0x7f7f7f7fu;
                if (part == 0) layout[256 + row] = nixl_gemm::ldExponents(sw + i);
            }
            asm volatile("fence.proxy.async;" ::: "memory"); // these generic-proxy writes are read by tcgen05.cp
            __syncwarp();
            if (lane == 0) mbarArriveClusterRelease(sffull0 + b * 8u);
            return true;
        };
        // Staging runs ahead of the issuer by up to two groups, across tile boundaries: the first groups of the next
        // tile are built before this tile's epilogue, so the issuer finds them waiting when the accumulator is free again.
        const int ahead = sf_groups < 2 ? sf_groups : 2;
        Tile cur, nxt;
        int ti = pair;
        bool have = tileAt(sh, p.groups, n_tiles, ti, cur);
        uint32_t g_base = 0;
        bool ok = true;
        if (have)
            for (int c = 0; c < ahead && ok; ++c) ok = stage(cur, c, g_base + c);
        for (int tile = 0; have && ok; ++tile) {
            for (int c = ahead; c < sf_groups && ok; ++c) ok = stage(cur, c, g_base + c);
            const bool have_next = tileAt(sh, p.groups, n_tiles, ti + pairs, nxt);
            if (have_next)
                for (int c = 0; c < ahead && ok; ++c) ok = stage(nxt, c, g_base + sf_groups + c);
            if (!ok) break;
            const Tile &t = cur;
            // Epilogue: this warp's 32 columns of D (TMEM lanes) for its half of the tokens (TMEM columns), up to
            // four blocks of 32.  All TMEM loads first, then the accumulator goes back to the issuer at once;
            // conversion and stores follow while the next tile's main loop is already running.
            if (!mbarWait(&sh.tmemFull, static_cast<uint32_t>(tile) & 1u, abort_flag)) break;
            tcFenceAfter();
            const int rows_t = sh.tileRows[t.g];
            const int half = (rows_t / 2 + 31) & ~31;
            const int first = part * half, mine = min(half, rows_t - first); // tokens of this warp (a multiple of 32, may be <= 0)
            float v[4][32];
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if (j * 32 < mine) tmemLoad32(lane_base + first + j * 32, v[j]);
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if (j * 32 < mine) tmemLoadWait(v[j]);
            tcFenceBefore();
            __syncwarp();
            if (lane == 0) mbarArriveCluster(tempty);
            const int local = t.mt * rows_t + first;
            const int left = min(mine, sh.rowCount[t.g] - local);
            __nv_bfloat16 *out = static_cast<__nv_bfloat16 *>(p.d) + (static_cast<long long>(sh.rowStart[t.g]) + local) * p.N + t.nt * (2 * BW) +
                static_cast<int>(cta) * BW + q * 32;
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if (j * 32 < left) storeCols32(v[j], out + static_cast<long long>(j * 32) * p.N, p.N, left - j * 32, lane);
            cur = nxt;
            have = have_next;
            ti += pairs;
            g_base += static_cast<uint32_t>(sf_groups);
        }
    }

    tcFenceBefore();
    __syncthreads();
    clusterSync();
    if (threadIdx.x == 0 && sh.abort) atomicOr(p.status, GEMM_ERR_TIMEOUT);
    if (warp == 2) {
        tcFenceAfter();
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols));
    }
}

} // namespace

cudaError_t nixl_gemm::launchMxPairKernel(const CUtensorMap &mapT, const CUtensorMap &mapT32, const CUtensorMap &mapT64, const CUtensorMap &mapW, const CUtensorMap &mapW2,
                                          const NixlGroupedGemmParams &p, cudaStream_t stream) {
    const size_t smem = size_t(kRingBytes) + size_t(2) * kSfBufBytes + sizeof(Shared) + 1024;
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    static bool attr_done[64] = {};
    static int max_pairs[64] = {};
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    attr[1] = nixl_pdl::overlapAttribute();
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    if (dev >= 0 && dev < 64 && !attr_done[dev]) {
        cudaError_t e = cudaFuncSetAttribute(groupedGemmMxPairKernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
        if (e != cudaSuccess) return e;
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        cfg.gridDim = dim3(static_cast<unsigned>(sms & ~1));
        int clusters = 0;
        e = cudaOccupancyMaxActiveClusters(&clusters, groupedGemmMxPairKernel, &cfg);
        if (e != cudaSuccess || clusters <= 0) {
            cudaGetLastError();
            clusters = sms / 2;
        }
        max_pairs[dev] = clusters;
        attr_done[dev] = true;
    }
    int pairs = (dev >= 0 && dev < 64) ? max_pairs[dev] : sms / 2;
    if (p.grid > 0 && p.grid / 2 < pairs) pairs = p.grid / 2 > 0 ? p.grid / 2 : 1;
    const long long max_tiles = (static_cast<long long>(p.a_rows + BT - 1) / BT + p.groups) * (p.N / (2 * BW));
    if (pairs > max_tiles) pairs = static_cast<int>(max_tiles);
    cfg.gridDim = dim3(static_cast<unsigned>(2 * pairs));
    cfg.numAttrs = 2;
    return cudaLaunchKernelEx(&cfg, groupedGemmMxPairKernel, mapT, mapT32, mapT64, mapW, mapW2, p);
}
