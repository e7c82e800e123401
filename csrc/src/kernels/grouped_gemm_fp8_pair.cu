// Grouped fp8 expert GEMM, 256 x 256 output tiles computed by CTA pairs (tcgen05 cta_group::2).
//
// Same math and operand formats as grouped_gemm_fp8.cu.  Two CTAs of a cluster share one tile:
// each loads its own 128 rows of A and 128 of the tile's 256 W rows per 128-channel step (32 KiB
// per CTA and step: half the L2 -> shared-memory traffic per MAC of 128 x 128 tiles), the even CTA
// issues M256 N256 K32 MMAs that read both CTAs' shared memory and write both CTAs' TMEM, and each
// CTA promotes and stores its own 128 rows.
//
// A 128-channel step is four MMAs into two neighbouring 128-column TMEM slots; two steps (four slots,
// all of TMEM) are in flight.  (Eight N = 128 instructions, one per slot, read A from shared memory twice and
// were slower by an eighth.)  A tile with at most 128 rows left runs as M = 128 (tailTile).
//
// What bounds this kernel is not the tensor pipe: four MMAs take 512 cycles, a step some 1100 (37 experts of 512 rows each, 2048 x
// 7168: 592 whole tiles, eight per pair; 350 us at 1.44 GHz under the power cap, tile ends counted in).  The promotion's own
// instructions are less than the MMAs' cycles too (128 two-wide FMAs per scheduler and step, and the TMEM reads), so what is not
// reached is their overlap: only two steps fit in TMEM and a slot is handed back late.  Uneven experts come on top: 16384 rows of 32
// experts take 305 us when all have 512 and 364 when they vary by an eighth.  Power is a bound beside these, not in front of them: the
// block-scaled kernel takes 246 and 281 us for the same products under the same cap.  What was done about the hand-offs:
//  * the issuing thread polls one barrier per step.  full[s] collects the producer's arrival (with
//    both CTAs' byte count) and one arrival from each of the pair's sixteen promotion warps, sent
//    when the warp has read the two slots the step will overwrite;
//  * that poll is a non-blocking test issued behind the previous step's MMAs: barrier instructions
//    in front of the MMAs delayed them by a few hundred cycles each;
//  * promotion warps poll once per step too (one commit covers both slots), arrive with relaxed
//    semantics (a cluster-scope release cost several hundred cycles per arrive) and fetch their
//    scales behind the arrive; they add with packed fp32 FMAs, half the instructions;
//  * ring positions are counters, not divisions, on the single-thread roles.
// (With W on the M side and tokens on the N side no rows are padded at all, but a token's scale then belongs to a register:
// reading the scales from shared memory, 4 bytes per lane and FMA, made a step twice as long.)
//
// Measured on one B200, back to back for half a second (that is, under the power cap), before / now: 31 experts that share
// 16384 rows unevenly, 2048 x 7168: 423 / 349 us (1.38 PFLOP/s); 32 experts, 32768 rows, 4096 x 4096: 844 / 713 us
// (1.54 PFLOP/s); one expert, 8192 rows, 4096 x 7168: 311 / 262 us (1.84 PFLOP/s).
//
//   warp 0      TMA producer (both CTAs; completion bytes are counted on the even CTA's barrier)
//   warp 1      MMA issuer (even CTA only); commits are multicast to both CTAs' barriers
//   warp 2      TMEM allocator (512 columns, cta_group::2)
//   warps 4-11  promotion + epilogue: lane quarter q = warp % 4, 64-column part (warp - 4) / 4 of
//               every slot; 128 fp32 accumulators per thread, so these warps raise their register
//               budget (setmaxnreg 232) with what the role warps give back (setmaxnreg 40; the two
//               budgets must leave the register file some slack, an exact fit never got its
//               increase granted)
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
using nixl_gemm::GEMM_ERR_ARRIVAL;
using nixl_gemm::GEMM_ERR_TIMEOUT;
using nixl_gemm::kMaxGroups;
using nixl_gemm::ldScale;
using nixl_gemm::waitArrivals;

constexpr int BM = 128;        // rows per CTA (256 per pair)
constexpr int BN = 256;        // tile columns
constexpr int BNS = 128;       // columns per TMEM slot: a step's accumulator is two neighbouring slots
constexpr int WROWS = 128;     // W rows each CTA keeps: the pair's MMA reads N = 256 rows, half from either CTA
constexpr int BK = 128;
constexpr int kStages = 6;
constexpr int kThreads = 384;
constexpr int kATileBytes = BM * BK;           // 16 KiB
constexpr int kStageBytes = kATileBytes + WROWS * BK; // 32 KiB per CTA
constexpr int kSlots = 4;
constexpr int kTmemCols = kSlots * BNS;        // 512
constexpr int kPromoWarps = 8;
// A step's full[] barrier collects the producer's arrival (which carries both CTAs' byte count) and
// one arrival from every promotion warp of the pair, sent when the warp has read the two TMEM
// slots the step is going to overwrite (the slots of the step two before it).
constexpr int kFullArrivals = 1 + 2 * kPromoWarps;

struct Shared {
    uint64_t full[kStages];       // used on the even CTA: a step may be issued (see kFullArrivals)
    uint64_t empty[kStages];      // per CTA: the MMAs that read the stage are done
    uint64_t tmemFull[2];         // per CTA: the two slots of an even / odd step are ready for promotion
    uint32_t tmemBase;
    int abort;
    int tilePrefix[kMaxGroups + 1];
    int rowStart[kMaxGroups];
    int rowCount[kMaxGroups];
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
// A whole 128-channel step of the issuer as one instruction sequence: four MMAs, two commits, and then a
// non-blocking test of the next step's barrier.  Barrier instructions placed in front of the MMAs
// delayed them by a few hundred cycles each, so the only poll of a step sits behind its MMAs, where
// the tensor pipe still has work queued.
__device__ __forceinline__ void issueKStep(uint32_t tmem_d, uint64_t da, uint64_t dw, uint32_t idesc, uint32_t bar_tmem_full, uint32_t bar_stage_empty,
                                           uint32_t peek_bar, uint32_t peek_par, uint32_t &ready_next) {
    asm volatile(
        "{\n"
        " .reg .pred pf, pacc, pnew;\n"
        " setp.ne.b32 pacc, %9, 0;\n"
        " setp.eq.b32 pnew, %9, 0;\n"
        " tcgen05.mma.cta_group::2.kind::f8f6f4 [%1], %2, %3, %4, {%10, %10, %10, %10, %10, %10, %10, %10}, pnew;\n"
        " add.u64 %2, %2, 2;\n add.u64 %3, %3, 2;\n"
        " tcgen05.mma.cta_group::2.kind::f8f6f4 [%1], %2, %3, %4, {%10, %10, %10, %10, %10, %10, %10, %10}, pacc;\n"
        " add.u64 %2, %2, 2;\n add.u64 %3, %3, 2;\n"
        " tcgen05.mma.cta_group::2.kind::f8f6f4 [%1], %2, %3, %4, {%10, %10, %10, %10, %10, %10, %10, %10}, pacc;\n"
        " add.u64 %2, %2, 2;\n add.u64 %3, %3, 2;\n"
        " tcgen05.mma.cta_group::2.kind::f8f6f4 [%1], %2, %3, %4, {%10, %10, %10, %10, %10, %10, %10, %10}, pacc;\n"
        " tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%5], %11;\n"
        " tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%6], %11;\n"
        " mbarrier.test_wait.parity.shared::cta.b64 pf, [%7], %8;\n"
        " selp.u32 %0, 1, 0, pf;\n"
        "}\n"
        : "=r"(ready_next), "+r"(tmem_d), "+l"(da), "+l"(dw)
        : "r"(idesc), "r"(bar_tmem_full), "r"(bar_stage_empty), "r"(peek_bar), "r"(peek_par), "r"(1u), "r"(0u), "h"(static_cast<uint16_t>(3))
        : "memory");
}

// D fp32, A and B e4m3, both K-major, M = m (256 or 128 rows of both CTAs together), N = 256.
__device__ __forceinline__ constexpr uint32_t instrDescPair(int m) {
    return (1u << 4) | (static_cast<uint32_t>(BN >> 3) << 17) | (static_cast<uint32_t>(m >> 4) << 24);
}

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

// A tile with at most 128 rows left runs as M = 128: 64 rows per CTA, and each CTA's TMEM lanes 0 - 63 hold their columns
// [0, 128) of the tile, lanes 64 - 127 the same rows' columns [128, 256).  Half the MMA time, half the promotion and half the
// A traffic of a tile whose second 128 rows would be padding.
__device__ __forceinline__ bool tailTile(const Shared &sh, const Tile &t) { return sh.rowCount[t.g] - t.mt * (2 * BM) <= BM; }

// Promotion of one tile: every step's sums leave TMEM, are scaled and added up in registers; then the tile is stored.  kTail: see
// tailTile (64 of 128 columns per thread; a loop of its own, as conditions in the full tile's loop made the compiler spill there).
// False when another role gave up.
template<bool kTail>
__device__ __forceinline__ bool promoteTile(Shared &sh, const float *sa_row, bool valid, bool fresh, const float *sw0, int k_steps, uint32_t lane_base, uint32_t full0, int lane,
                                            uint32_t &it, uint32_t &s2, bool &rdy, __nv_bfloat16 *out, long long row_stride, int rows_left) {
    volatile int *abort_flag = &sh.abort;
    constexpr int kBlocks = kTail ? 2 : 4; // of 32 columns
    const float *sw1 = kTail ? sw0 : sw0 + k_steps;
    uint64_t acc[kBlocks][16]; // fp32 pairs: left half's 64 columns, right half's
#pragma unroll
    for (int j = 0; j < kBlocks; ++j)
#pragma unroll
        for (int i = 0; i < 16; ++i) acc[j][i] = 0;
    // Scales are fetched two steps ahead and kept as loaded: multiplying them right away would make the warp
    // wait for the loads it has just issued.  (A loop unrolled over a ring of four made the compiler spill.)
    float a0 = valid ? ldScale(sa_row, fresh) : 0.f, w00 = ldScale(sw0, false), w10 = ldScale(sw1, false);
    float a1 = valid && k_steps > 1 ? ldScale(sa_row + 1, fresh) : 0.f, w01 = k_steps > 1 ? ldScale(sw0 + 1, false) : 0.f, w11 = k_steps > 1 ? ldScale(sw1 + 1, false) : 0.f;
#pragma unroll 1
    for (int ks = 0; ks < k_steps; ++ks, ++it) {
        const float s0 = a0 * w00, s1 = a0 * w10;
        const uint64_t s00 = pack2(s0, s0), s11 = pack2(s1, s1);
        a0 = a1;
        w00 = w01;
        w10 = w11;
        const int nxt = ks + 2;
        const uint32_t kp = it & 1u, sl = kp * 2u;
        if (!rdy && !mbarWait(&sh.tmemFull[kp], (it >> 1) & 1, abort_flag)) return false;
        tcFenceAfter();
        float v0[32], v1[32];
        tmemLoad32(lane_base + sl * BNS, v0);
        tmemLoad32(lane_base + sl * BNS + 32, v1);
        tmemLoadWait(v0);
        tmemLoadWait(v1);
        if constexpr (!kTail) {
            fmaScale32(acc[0], v0, s00);
            tmemLoad32(lane_base + (sl + 1) * BNS, v0); // second slot's loads run behind the first slot's FMAs
            fmaScale32(acc[1], v1, s00);
            tmemLoad32(lane_base + (sl + 1) * BNS + 32, v1);
        }
        // While those are in flight, look at the next step's barrier.
        rdy = mbarTest(&sh.tmemFull[kp ^ 1u], ((it + 1) >> 1) & 1);
        if constexpr (!kTail) {
            tmemLoadWait(v0);
            tmemLoadWait(v1);
        }
        // This step's slots are in registers: tell the step that reuses them.
        tcFenceBefore();
        __syncwarp();
        if (lane == 0) mbarArriveCluster(full0 + s2 * 8u);
        if (++s2 == kStages) s2 = 0;
        // The scale prefetch goes behind the arrive (loads issued before it would hold it up).
        if (nxt < k_steps) {
            a1 = valid ? ldScale(sa_row + nxt, fresh) : 0.f;
            w01 = ldScale(sw0 + nxt, false);
            if (!kTail) w11 = ldScale(sw1 + nxt, false);
        }
        fmaScale32(acc[kBlocks - 2], v0, kTail ? s00 : s11);
        fmaScale32(acc[kBlocks - 1], v1, kTail ? s00 : s11);
    }
    // Coalesced stores: see storeRows64.
    float lo[32], hi[32];
    unpack32(acc[0], lo);
    unpack32(acc[1], hi);
    storeRows64(lo, hi, out, row_stride, rows_left, lane);
    if constexpr (!kTail) {
        unpack32(acc[2], lo);
        unpack32(acc[3], hi);
        storeRows64(lo, hi, out + BNS, row_stride, rows_left, lane);
    }
    return true;
}

__global__ void __launch_bounds__(kThreads, 1)
groupedGemmPairKernel(const __grid_constant__ CUtensorMap mapA, const __grid_constant__ CUtensorMap mapA64, const __grid_constant__ CUtensorMap mapW, const NixlGroupedGemmParams p) {
    nixl_pdl::waitForPreviousKernel();
    extern __shared__ __align__(1024) unsigned char dyn[];
    unsigned char *tiles = reinterpret_cast<unsigned char *>((reinterpret_cast<uintptr_t>(dyn) + 1023) & ~uintptr_t(1023));
    Shared &sh = *reinterpret_cast<Shared *>(tiles + kStages * kStageBytes);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int n_tiles = p.N / BN, k_steps = p.K / BK;
    const uint32_t cta = clusterCtaRank(); // 0: issues the MMAs, 1: its partner
    const int pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;

    if (threadIdx.x == 0) {
        for (int s = 0; s < kStages; ++s) {
            mbarInit(&sh.full[s], kFullArrivals);
            mbarInit(&sh.empty[s], 1);
        }
        mbarInit(&sh.tmemFull[0], 1);
        mbarInit(&sh.tmemFull[1], 1);
        // The first two steps find their slots free: stand in for the promotion warps' arrivals.
        for (int s = 0; s < 2; ++s)
            asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0], %1;" ::"r"(smemU32(&sh.full[s])), "r"(2 * kPromoWarps) : "memory");
        sh.abort = 0;
        int run = 0;
        if (p.counts_flag) {
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
                next += c;
                run += ((c + 2 * BM - 1) / (2 * BM)) * n_tiles;
            }
            sh.tilePrefix[p.groups] = run;
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1 && !p.counts_flag) {
        int most;
        nixl_gemm::buildTileTable(p, n_tiles, [](int rows) { return (rows + 2 * BM - 1) / (2 * BM); }, sh.tilePrefix, sh.rowStart, sh.rowCount, most);
    }
    if (warp == 2) {
        // Both CTAs of the pair issue the paired allocation from the same warp and shared offset.
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smemU32(&sh.tmemBase)), "r"(kTmemCols));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;");
    }
    tcFenceBefore();
    __syncthreads();
    clusterSync(); // the partner's barriers exist before anything arrives on them
    tcFenceAfter();
    // With TMEM in hand: a kernel that moved in before could take it and then wait for this one.  (Not beside a dispatch.)
    if (!p.counts_flag && !p.disp_flag) nixl_pdl::allowNextKernel();
    const uint32_t tmem = sh.tmemBase;
    volatile int *abort_flag = &sh.abort;
    if (warp < 4) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 40;");
        if (warp == 0 && lane == 0) {
            // ------------------------------------------------------------ TMA producer (both CTAs)
            const uint32_t full0 = mapToCta(smemU32(&sh.full[0]), 0);
            uint32_t it = 0;
            Tile t;
            for (int ti = pair; tileAt(sh, p.groups, n_tiles, ti, t); ti += pairs) {
                const int rows_cta = tailTile(sh, t) ? BM / 2 : BM;
                const int lo = t.mt * (2 * BM) + static_cast<int>(cta) * rows_cta;
                const int row0 = sh.rowStart[t.g] + lo;
                const uint32_t bytes = static_cast<uint32_t>(2 * (rows_cta + WROWS) * BK); // both CTAs' shares
                if (p.disp_flag) {
                    waitArrivals(p, t.g, lo, min(lo + rows_cta, sh.rowCount[t.g]));
                    asm volatile("fence.proxy.async;" ::: "memory"); // peers' generic-proxy stores before our async-proxy reads
                }
                const int wrow = t.g * p.N + t.nt * BN + static_cast<int>(cta) * WROWS;
                for (int ks = 0; ks < k_steps; ++ks, ++it) {
                    const int s = it % kStages;
                    if (!mbarWait(&sh.empty[s], ((it / kStages) & 1) ^ 1, abort_flag)) goto role_done;
                    if (cta == 0) mbarExpectTx(&sh.full[s], bytes);
                    const uint32_t bar = full0 + static_cast<uint32_t>(s) * 8u;
                    unsigned char *st = tiles + s * kStageBytes;
                    tmaLoad2dPair(st, rows_cta == BM ? &mapA : &mapA64, ks * BK, row0, bar);
                    tmaLoad2dPair(st + kATileBytes, &mapW, ks * BK, wrow, bar);
                }
            }
        } else if (warp == 1 && lane == 0 && cta == 0) {
            // ------------------------------------------------------------ MMA issuer (even CTA)
            // One poll per four MMAs: full[s] completes when both CTAs' bytes have landed and all
            // promotion warps of the pair have read the step's two TMEM slots.
            uint32_t s = 0, full_par = 0, sl = 0; // ring positions as counters: no divisions on this thread
            uint32_t ready = 0;
            const uint32_t full_bar0 = smemU32(&sh.full[0]), empty_bar0 = smemU32(&sh.empty[0]), tfull_bar0 = smemU32(&sh.tmemFull[0]);
            const uint64_t desc0 = smemDesc(smemU32(tiles));
            Tile t;
            for (int ti = pair; tileAt(sh, p.groups, n_tiles, ti, t); ti += pairs) {
                const uint32_t idesc = instrDescPair(tailTile(sh, t) ? BM : 2 * BM);
                for (int ks = 0; ks < k_steps; ++ks) {
                    if (!ready && !mbarWait(&sh.full[s], full_par, abort_flag)) goto role_done;
                    tcFenceAfter();
                    uint32_t ns = s + 1, nfull_par = full_par;
                    if (ns == kStages) {
                        ns = 0;
                        nfull_par ^= 1u;
                    }
                    const uint64_t da = desc0 + static_cast<uint64_t>((s * kStageBytes) >> 4);
                    const uint64_t dw = da + static_cast<uint64_t>(kATileBytes >> 4);
                    issueKStep(tmem + sl * BNS, da, dw, idesc, tfull_bar0 + (sl >> 1) * 8u, empty_bar0 + s * 8u, full_bar0 + ns * 8u, nfull_par, ready);
                    sl ^= 2u;
                    s = ns;
                    full_par = nfull_par;
                }
            }
        }
    role_done:;
    } else {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 232;");
        // ---------------------------------------------------------------- promotion + epilogue
        const int q = warp & 3;
        const int part = (warp - 4) >> 2; // which 64 of a slot's 128 columns
        const uint32_t full0 = mapToCta(smemU32(&sh.full[0]), 0);
        const uint32_t lane_base = tmem + (static_cast<uint32_t>(q * 32) << 16) + part * 64;
        uint32_t it = 0;      // step counter, same numbering as the issuer's
        uint32_t s2 = 2;      // stage of step it + 2, the step that reuses this step's slots
        Tile t;
        const int n_blocks = p.N / 128;
        bool rdy = false;
        bool ok = true;
        for (int ti = pair; ok && tileAt(sh, p.groups, n_tiles, ti, t); ti += pairs) {
            const bool tail = tailTile(sh, t);
            // Full tile: one row, 64 columns of either half.  Tail: one of 64 rows, 64 columns of half q / 2.
            const int first_row = t.mt * (2 * BM) + (tail ? static_cast<int>(cta) * (BM / 2) + (q & 1) * 32 : static_cast<int>(cta) * BM + q * 32);
            const int local_row = first_row + lane;
            const bool valid = local_row < sh.rowCount[t.g];
            const bool fresh = p.disp_flag != nullptr; // the scales travel with the rows
            if (fresh) waitArrivals(p, t.g, first_row, min(first_row + 32, sh.rowCount[t.g]));
            const long long grow = static_cast<long long>(sh.rowStart[t.g]) + local_row;
            const float *sa_row = p.scale_a + grow * k_steps;
            const float *sw0 = p.scale_w + (static_cast<long long>(t.g) * n_blocks + t.nt * 2 + (tail ? q >> 1 : 0)) * k_steps;
            const int row8 = first_row + (lane & ~7);
            const int rows_left = sh.rowCount[t.g] - row8;
            __nv_bfloat16 *out = static_cast<__nv_bfloat16 *>(p.d) + (static_cast<long long>(sh.rowStart[t.g]) + row8) * p.N + t.nt * BN +
                (tail ? (q >> 1) * BNS : 0) + part * 64 + (lane & 7) * 8;
            ok = tail ? promoteTile<true>(sh, sa_row, valid, fresh, sw0, k_steps, lane_base, full0, lane, it, s2, rdy, out, p.N, rows_left)
                      : promoteTile<false>(sh, sa_row, valid, fresh, sw0, k_steps, lane_base, full0, lane, it, s2, rdy, out, p.N, rows_left);
        }
    }

    // Neither CTA may leave (or free TMEM) while its partner can still read its shared memory,
    // write its TMEM or arrive on its barriers.
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

cudaError_t nixl_gemm::launchPairKernel(const CUtensorMap &mapA, const CUtensorMap &mapA64, const CUtensorMap &mapW, const NixlGroupedGemmParams &p, cudaStream_t stream) {
    const size_t smem = size_t(kStages) * kStageBytes + sizeof(Shared) + 1024;
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
        cudaError_t e = cudaFuncSetAttribute(groupedGemmPairKernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
        if (e != cudaSuccess) return e;
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        // How many pairs can be resident at once: a persistent grid must not exceed it.
        cfg.gridDim = dim3(static_cast<unsigned>(sms & ~1));
        int clusters = 0;
        e = cudaOccupancyMaxActiveClusters(&clusters, groupedGemmPairKernel, &cfg);
        if (e != cudaSuccess || clusters <= 0) {
            cudaGetLastError();
            clusters = sms / 2;
        }
        max_pairs[dev] = clusters;
        attr_done[dev] = true;
    }
    int pairs = (dev >= 0 && dev < 64) ? max_pairs[dev] : sms / 2;
    if (p.grid > 0 && p.grid / 2 < pairs) pairs = p.grid / 2 > 0 ? p.grid / 2 : 1;
    const long long max_tiles = (static_cast<long long>(p.a_rows + 2 * BM - 1) / (2 * BM) + p.groups) * (p.N / BN);
    if (pairs > max_tiles) pairs = static_cast<int>(max_tiles);
    cfg.gridDim = dim3(static_cast<unsigned>(2 * pairs));
    cfg.numAttrs = p.counts_flag || p.disp_flag ? 1 : 2; // (one that waits for a dispatch on another stream: not before the stream's own turn)
    return cudaLaunchKernelEx(&cfg, groupedGemmPairKernel, mapA, mapA64, mapW, p);
}
