// MoE expert-parallel dispatch / combine for one NVLink domain (contract and algorithm:
// include/kernels/nixl_kernels.h).
//
// All are persistent grids of 256 threads, launched cooperatively where they contain a grid barrier (every CTA resident,
// so that it cannot deadlock).  Peer memory is reached through the remote memory view prepared by the agent: plain stores
// over NVLink, release-ordered flags, and bounded waits that mask a silent peer instead of hanging the GPU.
#include <cooperative_groups.h>
#include <cuda_bf16.h>
#include <cuda_fp8.h>
#include <cuda_runtime.h>

#include "device/nixl_device_layout.h"
#include "kernels/nixl_kernels.h"
#include "kernels/programmatic_launch.cuh"

namespace {

constexpr int kThreads = 256;
constexpr int kMaxRanks = 64;
constexpr int kMaxTopk = 16;
constexpr int kGroup = 128; // channels per quantisation group

enum : int { ST_PEER_TIMEOUT = 1, ST_BARRIER_TIMEOUT = 2, ST_CAPACITY = 4 };

// ------------------------------------------------------------------ small device helpers

__device__ __forceinline__ uint64_t nowNs() {
    uint64_t t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
    return t;
}
__device__ __forceinline__ uint64_t ldAcquireSys(const uint64_t *p) {
    uint64_t v;
    asm volatile("ld.acquire.sys.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void stReleaseSys(uint64_t *p, uint64_t v) {
    asm volatile("st.release.sys.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
__device__ __forceinline__ void stReleaseGpu(uint64_t *p, uint64_t v) {
    asm volatile("st.release.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
__device__ __forceinline__ unsigned addAcqRelGpu(unsigned *p, unsigned v) {
    unsigned old;
    asm volatile("atom.add.acq_rel.gpu.global.u32 %0, [%1], %2;" : "=r"(old) : "l"(p), "r"(v) : "memory");
    return old;
}
__device__ __forceinline__ int addAcqRelSys(int *p, int v) {
    int old;
    asm volatile("atom.add.acq_rel.sys.global.s32 %0, [%1], %2;" : "=r"(old) : "l"(p), "r"(v) : "memory");
    return old;
}
__device__ __forceinline__ unsigned ldAcquireGpu(const unsigned *p) {
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ int ldVolatile(const int *p) { return *reinterpret_cast<const volatile int *>(p); }
// Rows are loaded coherently, past L1: not through the read-only path, which is for data that nobody writes while the kernel runs.
// The kernel in front of an overlapped launch still writes them then, and so do peers whose flag this kernel waits for.
__device__ __forceinline__ uint4 ldStream16(const void *p) {
    uint4 v;
    asm volatile("ld.global.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
    return v;
}
__device__ __forceinline__ void stPeer16(void *p, const uint4 &v) {
    asm volatile("st.global.L1::no_allocate.v4.u32 [%0], {%1,%2,%3,%4};" ::"l"(p), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}

// 32 bytes as two 16-byte halves; one access where the address allows.
__device__ __forceinline__ void ldStream32(const void *p, bool wide, uint4 &lo, uint4 &hi) {
    if (wide) {
        asm volatile("ld.global.L1::no_allocate.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                     : "=r"(lo.x), "=r"(lo.y), "=r"(lo.z), "=r"(lo.w), "=r"(hi.x), "=r"(hi.y), "=r"(hi.z), "=r"(hi.w)
                     : "l"(p));
    } else {
        lo = ldStream16(p);
        hi = ldStream16(static_cast<const char *>(p) + 16);
    }
}
__device__ __forceinline__ void stPeer32(void *p, bool wide, const uint4 &lo, const uint4 &hi) {
    if (wide) {
        asm volatile("st.global.L1::no_allocate.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(p), "r"(lo.x), "r"(lo.y), "r"(lo.z), "r"(lo.w), "r"(hi.x),
                     "r"(hi.y), "r"(hi.z), "r"(hi.w)
                     : "memory");
    } else {
        stPeer16(p, lo);
        stPeer16(static_cast<char *>(p) + 16, hi);
    }
}

__device__ __forceinline__ char *peerBase(const void *view, int r) {
    const nixlMemViewEntry *e = reinterpret_cast<const nixlMemViewEntry *>(static_cast<const char *>(view) + sizeof(nixlMemViewHeader));
    return reinterpret_cast<char *>(e[r].ptr);
}

// Waits until *flag >= epoch.  False on timeout.
__device__ __forceinline__ bool waitFlag(const uint64_t *flag, uint64_t epoch, uint64_t timeout_ns) {
    uint64_t t0 = 0;
    unsigned spins = 0;
    while (ldAcquireSys(flag) < epoch) {
        if ((++spins & 31u) == 0) {
            const uint64_t now = nowNs();
            if (t0 == 0) t0 = now;
            else if (now - t0 > timeout_ns) return false;
        }
    }
    return true;
}

// Grid-wide barrier on two words {arrivals, generation}.  Bounded: on timeout sets the status
// bit and returns (the caller's results are then unreliable, which the host sees in `status`).
__device__ __forceinline__ void gridBarrier(unsigned *bar, int *status, uint64_t timeout_ns) {
    __syncthreads();
    if (threadIdx.x == 0) {
        const unsigned gen = ldAcquireGpu(bar + 1);
        __threadfence();
        if (atomicAdd(bar, 1u) == gridDim.x - 1) {
            bar[0] = 0;
            __threadfence();
            atomicAdd(bar + 1, 1u);
        } else {
            uint64_t t0 = 0;
            unsigned spins = 0;
            while (ldAcquireGpu(bar + 1) == gen) {
                if ((++spins & 63u) == 0) {
                    const uint64_t now = nowNs();
                    if (t0 == 0) t0 = now;
                    else if (now - t0 > timeout_ns) {
                        atomicOr(status, ST_BARRIER_TIMEOUT);
                        break;
                    }
                }
            }
        }
    }
    __syncthreads();
}

// The same for a kernel whose last CTA sets the word back to zero when all have left: one operation to arrive, no generation to read.
// The word stays raised until then, so nothing else may use it: a combine of the same buffer may run on another stream meanwhile.
__device__ __forceinline__ void gridBarrierOnce(unsigned *bar, int *status, uint64_t timeout_ns) {
    __syncthreads();
    if (threadIdx.x == 0 && addAcqRelGpu(bar, 1u) + 1 < gridDim.x) {
        uint64_t t0 = 0;
        unsigned spins = 0;
        while (ldAcquireGpu(bar) < gridDim.x) {
            if ((++spins & 63u) == 0) {
                const uint64_t now = nowNs();
                if (t0 == 0) t0 = now;
                else if (now - t0 > timeout_ns) {
                    atomicOr(status, ST_BARRIER_TIMEOUT);
                    break;
                }
            }
        }
    }
    __syncthreads();
}

// Threads cooperating on one token / row: as many as keeps the whole grid busy, a power of two
// between one warp and one CTA.
__device__ __forceinline__ int threadsPerItem(long long items) {
    const long long avail = static_cast<long long>(gridDim.x) * kThreads;
    int t = kThreads;
    while (t > 32 && static_cast<long long>(t) * items > avail) t >>= 1;
    return t;
}

// ------------------------------------------------------------------ dispatch

// Quantises one 128-channel group held by 8 lanes (16 bf16 each): returns 16 e4m3 bytes and the
// group's scale, the same in the eight lanes.
__device__ __forceinline__ uint4 quantGroup(const uint4 &lo, const uint4 &hi, bool round_scale, float &scale_out) {
    const __nv_bfloat162 *hl = reinterpret_cast<const __nv_bfloat162 *>(&lo), *hh = reinterpret_cast<const __nv_bfloat162 *>(&hi);
    float f[16];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float2 a = __bfloat1622float2(hl[i]), b = __bfloat1622float2(hh[i]);
        f[2 * i] = a.x;
        f[2 * i + 1] = a.y;
        f[8 + 2 * i] = b.x;
        f[8 + 2 * i + 1] = b.y;
    }
    float amax = 0.f;
#pragma unroll
    for (int i = 0; i < 16; ++i) amax = fmaxf(amax, fabsf(f[i]));
#pragma unroll
    for (int o = 4; o >= 1; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
    amax = fmaxf(amax, 1e-4f); // margin of the reference's cast (csrc/kernels/utils.cuh:430-456): never divide by ~0
    float scale = amax / 448.f, inv;
    if (round_scale) {
        const int ex = static_cast<int>(ceilf(log2f(scale)));
        scale = exp2f(static_cast<float>(ex));
        inv = exp2f(static_cast<float>(-ex));
    } else {
        inv = 448.f / amax;
    }
    scale_out = scale;
    uint32_t w[8];
#pragma unroll
    for (int i = 0; i < 8; ++i)
        w[i] = static_cast<uint32_t>(__nv_cvt_float2_to_fp8x2(make_float2(f[2 * i] * inv, f[2 * i + 1] * inv), __NV_SATFINITE, __NV_E4M3));
    return make_uint4(w[0] | (w[1] << 16), w[2] | (w[3] << 16), w[4] | (w[5] << 16), w[6] | (w[7] << 16));
}

// Dispatch.  Every CTA owns a contiguous range of tokens.  It counts its copies per expert in shared memory and adds them to
// the rank's counters with one atomic per expert, whose old value is at the same time this CTA's place among the rank's rows of
// that expert: there is no atomic, and no wait, per copy.  (One per copy on E counters, to count, to reserve a row and to
// report it sent, and a staging buffer per token that left room for eight warps per SM in bf16, was what bounded it.)
// In the data phase a warp takes a token or a part of one (slices of 512 channels), reads 32 bytes per lane, quantises in
// registers and stores to the up to K receivers; nothing is staged and warps do not wait for each other, so it is bound by
// the stores.  With few tokens it is a chain of latencies (counters, grid barrier, exchange of counts, tables, rows, flags),
// which is why nothing in it is read or fenced twice; a group of one rank takes its counts from the grid barrier instead of
// through its own flags.
// Measured on one B200, one rank, 32 experts, top-8, before / now: 4096 tokens x 7168 bf16 131 / 113 us (528 MB, 4.7 TB/s; the
// rows written, 470 MB, are the bound), fp8 97 / 73 us, 4096 x 4096 fp8 74 / 47 us (3.6 TB/s); 128 tokens x 7168 fp8, low-latency
// layout 21.6 / 13.4 us (8.4 with fixed places); 1 token 20.5 / 11.9 us (7.8).
// A group of one rank then dropped what only others need (flags early, rows counted as sent), except in the launch that a GEMM
// beside it follows row by row; every group reads the routing once, arrives at the grid barrier with one operation and calls its
// rows into L2 while it counts.  Compact layout, 32 experts, top-8, us before / after: 1 token 17.9 / 11.0, 300 x 4096 bf16 18.1 /
// 15.5, 700 29.5 / 19.8, 1500 40.3 / 32.0; 4096 x 4096 with power-of-two scales 47.2 / 39.8, 4096 x 7168 bf16 116 / 114 (bound by
// the writes to some 4700 rows that are open at a time).
constexpr int kBatch = 32;  // tokens whose rows are looked up together, and reported as sent together
constexpr int kSlices = 2;  // slices of a token in flight per warp: 2 KiB
constexpr int kDispatchCtas = 4; // per SM, with many tokens
constexpr int kPrefetch = 8;     // tokens of a CTA that are called into L2 while the copies are counted (58 MB of 4096 x 7168)

// Shared memory of the dispatch: `tables` words per expert and the batch's rows.  Where three tables do not fit (above some
// 19,000 experts) the rank's totals stay in global memory; two tables hold 28,000.
constexpr size_t kDispatchSmemMax = 226 * 1024;
__host__ __device__ __forceinline__ size_t dispatchSmem(int E, int K, int tables) {
    return size_t(tables) * E * sizeof(int) + size_t(kBatch) * K * (sizeof(int) + 1) + 16;
}
__host__ __device__ __forceinline__ int dispatchTables(int E, int K) { return dispatchSmem(E, K, 3) <= kDispatchSmemMax ? 3 : 2; }

__host__ __device__ __forceinline__ bool placesAreFixed(const NixlEpDispatchParams &p) { return p.R == 1 && p.rows_per_expert > 0 && p.phases == 3; }

template<bool kFp8> __device__ __forceinline__ void dispatchTokens(const NixlEpDispatchParams &p, const int *rows, const unsigned char *dests, char *const *peer_sh,
                                                                   long long t0, int n_tokens, int parts) {
    const int groups = p.H / kGroup, slices = p.H / 512;
    const int row_bytes = kFp8 ? p.H : p.H * 2;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const char *x = static_cast<const char *>(p.x);
    const bool wide_in = (reinterpret_cast<uintptr_t>(x) & 31) == 0; // rows are multiples of 1 KiB
    const bool round_scale = (p.round_scale | p.use_ue8m0) != 0;
    for (int item = warp; item < n_tokens * parts; item += kThreads / 32) {
        const int tl = item / parts, part = item - tl * parts;
        const long long t = t0 + tl;
        // Lane k < K: where the token's k-th copy goes.
        long long row = -1;
        char *peer = nullptr;
        int dest = -1;
        if (lane < p.K) {
            row = rows[tl * p.K + lane];
            dest = dests[tl * p.K + lane];
            peer = peer_sh[dest];
        }
        const char *src = x + t * p.H * 2 + lane * 32;
        char *to = row >= 0 ? peer + p.lay.off_recv_x + row * row_bytes : nullptr;
        char *to_scales = row >= 0 ? peer + p.lay.off_recv_scales + row * groups * (p.use_ue8m0 ? 1 : 4) : nullptr;
        const int s_end = slices * (part + 1) / parts; // this part's slices are consecutive: runs of a few KiB at every receiver
        for (int s0 = slices * part / parts; s0 < s_end; s0 += kSlices) {
            uint4 lo[kSlices], hi[kSlices];
#pragma unroll
            for (int j = 0; j < kSlices; ++j) ldStream32(src + static_cast<long long>(min(s0 + j, s_end - 1)) * 1024, wide_in, lo[j], hi[j]); // (past the end: the last slice again, not stored)
            float4 sc = make_float4(0.f, 0.f, 0.f, 0.f); // lane j: the four scales of slice j
            if constexpr (kFp8) {
#pragma unroll
                for (int j = 0; j < kSlices; ++j) {
                    float scale;
                    lo[j] = quantGroup(lo[j], hi[j], round_scale, scale);
                    const float4 f = make_float4(__shfl_sync(0xffffffffu, scale, 0), __shfl_sync(0xffffffffu, scale, 8), __shfl_sync(0xffffffffu, scale, 16),
                                                 __shfl_sync(0xffffffffu, scale, 24));
                    if (lane == j) sc = f;
                }
            }
            const int my_slice = s0 + lane; // whose scales this lane stores
            // A power-of-two scale is its exponent: one biased byte per group, four groups per word.
            const uint32_t exps = ((__float_as_uint(sc.x) >> 23) & 0xffu) | (((__float_as_uint(sc.y) >> 23) & 0xffu) << 8) |
                (((__float_as_uint(sc.z) >> 23) & 0xffu) << 16) | (((__float_as_uint(sc.w) >> 23) & 0xffu) << 24);
            for (int k = 0; k < p.K; ++k) {
                char *dst = reinterpret_cast<char *>(__shfl_sync(0xffffffffu, reinterpret_cast<unsigned long long>(to), k));
                if (dst == nullptr) continue; // uniform
                const bool wide_out = (reinterpret_cast<uintptr_t>(dst) & 31) == 0;
#pragma unroll
                for (int j = 0; j < kSlices; ++j) {
                    const int s = s0 + j;
                    if (s >= s_end) break;
                    if constexpr (kFp8) stPeer16(dst + s * 512 + lane * 16, lo[j]);
                    else stPeer32(dst + s * 1024 + lane * 32, wide_out, lo[j], hi[j]);
                }
                if constexpr (kFp8) {
                    char *ds = reinterpret_cast<char *>(__shfl_sync(0xffffffffu, reinterpret_cast<unsigned long long>(to_scales), k));
                    if (lane < kSlices && my_slice < s_end) {
                        if (p.use_ue8m0) *reinterpret_cast<uint32_t *>(ds + my_slice * 4) = exps;
                        else *reinterpret_cast<float4 *>(ds + my_slice * 16) = sc;
                    }
                }
            }
        }
        if (part != 0) continue;
        if (row >= 0) *reinterpret_cast<uint2 *>(peer + p.lay.off_recv_info + row * 8) = make_uint2(static_cast<unsigned>(p.rank), static_cast<unsigned>(t * p.K + lane));
        // Group record of this token for every rank that got copies of it (lane d serves rank d): the rows
        // and their weights, tagged with the step number so that what an earlier step left in the slot
        // is never taken for new.  Ranks without a copy get nothing; their slot keeps an old tag.
        if (p.topk_weights != nullptr) {
            const float weight = lane < p.K ? p.topk_weights[t * p.K + lane] : 0.f;
            int n = 0;
            int rec_rows[8] = {0, 0, 0, 0, 0, 0, 0, 0};
            uint32_t rec_w[8] = {0, 0, 0, 0, 0, 0, 0, 0};
            for (int k = 0; k < p.K; ++k) { // K <= 8 here
                const int rk = __shfl_sync(0xffffffffu, static_cast<int>(row), k), dk = __shfl_sync(0xffffffffu, dest, k);
                const uint32_t wk = __float_as_uint(__shfl_sync(0xffffffffu, weight, k));
                if (rk < 0 || dk != lane) continue;
#pragma unroll
                for (int i = 0; i < 8; ++i)
                    if (i == n) {
                        rec_rows[i] = rk;
                        rec_w[i] = wk;
                    }
                ++n;
            }
            if (n > 0) { // lane is a rank that holds copies
                uint4 *dst = reinterpret_cast<uint4 *>(peer_sh[lane] + p.lay.off_grp) + (static_cast<long long>(p.rank) * p.max_tokens + t) * 5;
                stPeer16(dst, make_uint4(static_cast<unsigned>(n), static_cast<unsigned>(p.epoch & 0x7fffffffull), 0u, 0u));
                stPeer16(dst + 1, make_uint4(rec_rows[0], rec_rows[1], rec_rows[2], rec_rows[3]));
                stPeer16(dst + 2, make_uint4(rec_rows[4], rec_rows[5], rec_rows[6], rec_rows[7]));
                stPeer16(dst + 3, make_uint4(rec_w[0], rec_w[1], rec_w[2], rec_w[3]));
                stPeer16(dst + 4, make_uint4(rec_w[4], rec_w[5], rec_w[6], rec_w[7]));
            }
        }
    }
}

template<bool kKeepTotals> // the rank's totals fit into shared memory
__global__ void __launch_bounds__(kThreads, kDispatchCtas) epDispatchKernel(const __grid_constant__ NixlEpDispatchParams p) {
    extern __shared__ __align__(16) unsigned char smem[];
    // (A launch that waits for peers, or only receives, lets nothing in: see programmatic_launch.cuh.)
    if (p.R == 1 && (p.phases & 1)) nixl_pdl::allowNextKernel();
    nixl_pdl::waitForPreviousKernel();
    const int El = p.E / p.R;
    // shared: place[E] | mine[E] | total[E] (kKeepTotals) | rows[kBatch * K] | dests[kBatch * K]
    int *place = reinterpret_cast<int *>(smem); // row of this CTA's next copy to expert e at its receiver
    int *mine = place + p.E;                    // this CTA's copies per expert: of its whole range, then of a batch
    int *ebase = mine;                          // in between: first row of expert e at its receiver
    int *total = mine + p.E;                    // the rank's copies per expert (all CTAs')
    int *rows = kKeepTotals ? total + p.E : total;
    auto totalOf = [&](int e) { return kKeepTotals ? total[e] : ldVolatile(p.scr.cnt + e); }; // (behind the grid barrier)
    unsigned char *dests = reinterpret_cast<unsigned char *>(rows + kBatch * p.K);

    char *self = peerBase(p.peers, p.rank);
    const int tid = threadIdx.x;
    __shared__ char *peer_sh[kMaxRanks]; // the data phase looks a peer up per row: keep the table on chip
    __shared__ int masked[kMaxRanks];
    if (tid < p.R) {
        peer_sh[tid] = peerBase(p.peers, tid);
        masked[tid] = ldVolatile(p.scr.mask + tid);
    }
    // One rank, low-latency layout, send and receive in one launch: a row's place is known without anybody's counts (expert e
    // starts at e * rows_per_expert, the CTA's share at what its atomic returned), so nothing is waited for; the last CTA
    // out publishes the counts.  13.4 -> 8.4 us for 128 tokens x 7168, 11.9 -> 7.8 us for one token.
    const bool fixed = placesAreFixed(p);
    const long long t_first = static_cast<long long>(p.T) * blockIdx.x / gridDim.x, t_end = static_cast<long long>(p.T) * (blockIdx.x + 1) / gridDim.x;
    // A group of one rank that sends in this launch has everybody's counts, its own, from the grid barrier, and sends every
    // row itself, so it waits for no flag.  (A launch that only receives waits for the flags like any other: the caller may have
    // sent on another stream.)  Unless a GEMM beside this launch takes the rows as they arrive (bit 2 of the phases), it also counts
    // no rows as sent, and the last CTA out raises all flags.
    const bool own = p.R == 1 && (p.phases & 1);
    const bool flags_last = own && !(p.phases & 4);

    if (p.phases & 1) {
        // 1. this CTA's copies per expert, and its place among the rank's
        const int n_copies = static_cast<int>(t_end - t_first) * p.K;
        for (int at = tid * 128; at < min(static_cast<int>(t_end - t_first), kPrefetch) * p.H * 2; at += kThreads * 128)
            asm volatile("prefetch.global.L2 [%0];" ::"l"(static_cast<const char *>(p.x) + t_first * p.H * 2 + at));
        for (int e = tid; e < p.E; e += kThreads) mine[e] = 0;
        __syncthreads();
        for (int i = tid; i < n_copies; i += kThreads) {
            const long long e = p.topk_idx[t_first * p.K + i];
            const bool valid = e >= 0 && e < p.E;
            if (valid && masked[static_cast<int>(e) / El] == 0) atomicAdd(mine + e, 1);
            if (i < kBatch * p.K) rows[i] = valid ? static_cast<int>(e) : -1; // (the first batch's experts: read once)
        }
        __syncthreads();
        for (int e = tid; e < p.E; e += kThreads) {
            place[e] = mine[e] ? atomicAdd(p.scr.cnt + e, mine[e]) : 0;
            if (fixed) place[e] += e * p.rows_per_expert;
        }
        if (fixed) __syncthreads();
    }
    if ((p.phases & 1) && !fixed) {
        gridBarrierOnce(p.scr.barrier + 3, p.scr.status, p.timeout_ns);
        for (int e = tid; e < p.E && kKeepTotals; e += kThreads) total[e] = ldVolatile(p.scr.cnt + e);
        __syncthreads();

        // 2. all-gather of counts: CTA b serves destination ranks b, b+grid, ...
        for (int d = blockIdx.x; d < p.R; d += gridDim.x) {
            char *peer = peer_sh[d];
            if (masked[d] != 0 || peer == nullptr) continue;
            int *dst = reinterpret_cast<int *>(peer + p.lay.off_counts) + static_cast<long long>(p.rank) * p.E;
            for (int e = tid; e < p.E; e += kThreads) dst[e] = totalOf(e);
            if (tid == 0) reinterpret_cast<int *>(peer + p.lay.off_grp_tokens)[p.rank] = p.topk_weights != nullptr ? p.T : 0;
            // Experts of that rank that get nothing from us are complete right away.
            if (flags_last) break;
            uint64_t *dflag = reinterpret_cast<uint64_t *>(peer + p.lay.off_disp_flag);
            __syncthreads(); // the release below covers the whole CTA's stores
            if (tid == 0) stReleaseSys(reinterpret_cast<uint64_t *>(peer + p.lay.off_counts_flag) + p.rank, p.epoch);
            for (int le = tid; le < El; le += kThreads)
                if (totalOf(d * El + le) == 0) stReleaseSys(dflag + static_cast<long long>(le) * p.R + p.rank, p.epoch);
        }
    }

    // 3. wait for everybody's counts (every CTA looks for itself: 8 flags, no grid barrier needed)
    if (!fixed) {
        const uint64_t *cflag = reinterpret_cast<const uint64_t *>(self + p.lay.off_counts_flag);
        if (tid < p.R) {
            if (masked[tid] == 0 && peer_sh[tid] != nullptr) {
                if (!own && !waitFlag(cflag + tid, p.epoch, p.timeout_ns)) {
                    atomicExch(p.scr.mask + tid, 1);
                    atomicOr(p.scr.status, ST_PEER_TIMEOUT);
                }
            } else if (peer_sh[tid] == nullptr) {
                atomicExch(p.scr.mask + tid, 1);
            }
            if (!own) masked[tid] = ldVolatile(p.scr.mask + tid);
        }
        __syncthreads();

        // 4. placement tables.  counts[r][e] is the local copy of the all-gather.
        const int *counts = reinterpret_cast<const int *>(self + p.lay.off_counts);
        for (int e = tid; e < p.E; e += kThreads) {
            int b = 0, all = 0;
            for (int r = 0; r < p.R; ++r) {
                const int c = own ? totalOf(e) : ldVolatile(counts + static_cast<long long>(r) * p.E + e); // (loads of all ranks in flight together)
                if (masked[r] != 0) continue;
                if (r < p.rank) b += c;
                all += c;
            }
            if (p.phases & 1) place[e] += b;
            ebase[e] = all; // totals first, turned into per-rank prefixes below
        }
        __syncthreads();
        if (p.rows_per_expert > 0) {
            for (int e = tid; e < p.E; e += kThreads)
                if (ebase[e] > p.rows_per_expert) atomicOr(p.scr.status, ST_CAPACITY);
            __syncthreads();
            for (int e = tid; e < p.E; e += kThreads) ebase[e] = (e % El) * p.rows_per_expert;
        } else {
            // exclusive prefix over the local experts of a destination rank, a warp per rank
            const int lane = tid & 31;
            for (int r = tid >> 5; r < p.R; r += kThreads / 32) {
                int run = 0;
                for (int l0 = 0; l0 < El; l0 += 32) {
                    const int c = l0 + lane < El ? ebase[r * El + l0 + lane] : 0;
                    int upto = c;
#pragma unroll
                    for (int o = 1; o < 32; o <<= 1) {
                        const int below = __shfl_up_sync(0xffffffffu, upto, o);
                        if (lane >= o) upto += below;
                    }
                    if (l0 + lane < El) ebase[r * El + l0 + lane] = run + upto - c;
                    run += __shfl_sync(0xffffffffu, upto, 31);
                }
                if (lane == 0 && run > p.cap) atomicOr(p.scr.status, ST_CAPACITY);
            }
        }
        __syncthreads();

        // Receiver-side bookkeeping is known as soon as the counts are: CTA 0 publishes it.
        if (blockIdx.x == 0 && (p.phases & 6)) {
            for (int le = tid; le < El; le += kThreads) {
                const int e = p.rank * El + le;
                int all = 0;
                for (int r = 0; r < p.R; ++r) {
                    int c = own ? totalOf(e) : ldVolatile(counts + static_cast<long long>(r) * p.E + e);
                    if (masked[r] != 0) c = 0;
                    p.layout_range[static_cast<long long>(le) * p.R + r] = (static_cast<long long>(all) << 32) | static_cast<unsigned>(c);
                    all += c;
                }
                p.recv_count[le] = all;
                p.expert_offsets[le] = ebase[e];
                if (le == El - 1) p.expert_offsets[El] = ebase[e] + (p.rows_per_expert > 0 ? p.rows_per_expert : all);
            }
        }
        if (p.phases & 1)
            for (int e = tid; e < p.E; e += kThreads) place[e] += ebase[e];
        __syncthreads(); // the first batch puts its counts where the first rows are
    }

    if (p.phases & 1) {
        // 5. data, a batch of tokens at a time
        const int n_mine = static_cast<int>(t_end - t_first);
        // Parts of a token that warps share: enough for two items per warp, so that the last round is not nearly empty.
        int parts = 1;
        while (parts < 8 && 2 * parts <= p.H / 512 && n_mine * parts < 2 * (kThreads / 32)) parts <<= 1;
        for (long long tb = t_first; tb < t_end; tb += kBatch) {
            const int n = static_cast<int>(t_end - tb < kBatch ? t_end - tb : kBatch);
            for (int e = tid; e < p.E; e += kThreads) mine[e] = 0;
            __syncthreads();
            for (int i = tid; i < n * p.K; i += kThreads) {
                int e = rows[i];
                if (tb != t_first) {
                    const long long wide = p.topk_idx[tb * p.K + i];
                    e = wide >= 0 && wide < p.E ? static_cast<int>(wide) : -1;
                }
                int row = -1, dest = 0;
                if (e >= 0 && masked[e / El] == 0) {
                    dest = e / El;
                    row = atomicAdd(place + e, 1);
                    if (row >= p.cap) row = -1; // flagged as ST_CAPACITY above
                    atomicAdd(mine + e, 1);     // counted as sent even then
                }
                rows[i] = row;
                dests[i] = static_cast<unsigned char>(dest);
                if (p.send_row != nullptr) p.send_row[tb * p.K + i] = row;
            }
            __syncthreads();
            if (p.use_fp8) dispatchTokens<true>(p, rows, dests, peer_sh, tb, n, parts);
            else dispatchTokens<false>(p, rows, dests, peer_sh, tb, n, parts);
            __syncthreads(); // all stores of the batch issued (and its tables free for the next one)
            // Count the batch's rows as sent.  Whoever completes an expert's rows raises that expert's arrival flag at its rank.
            for (int e = tid; e < p.E && !flags_last; e += kThreads) {
                const int c = mine[e];
                if (c == 0) continue;
                // One operation releases this CTA's rows and acquires the other CTAs'.
                const int done = addAcqRelSys(p.scr.sent + e, c) + c;
                if (done == totalOf(e)) stReleaseSys(reinterpret_cast<uint64_t *>(peer_sh[e / El] + p.lay.off_disp_flag) + static_cast<long long>(e % El) * p.R + p.rank, p.epoch);
            }
        }
    }

    if ((p.phases & 2) && !own) {
        // 6. arrivals: El x R flags, spread over the grid's threads
        const uint64_t *dflag = reinterpret_cast<const uint64_t *>(self + p.lay.off_disp_flag);
        const int nflags = El * p.R;
        for (int i = blockIdx.x * kThreads + tid; i < nflags; i += gridDim.x * kThreads) {
            const int r = i % p.R;
            if (ldVolatile(p.scr.mask + r) != 0) continue;
            if (!waitFlag(dflag + i, p.epoch, p.timeout_ns)) {
                atomicExch(p.scr.mask + r, 1);
                atomicOr(p.scr.status, ST_PEER_TIMEOUT);
            }
        }
    }

    // 7. the last CTA out leaves the scratch counters at zero for the next call (nobody waits for it)
    if (p.phases & 1) {
        __shared__ int last;
        __syncthreads();
        if (tid == 0) { // releases this CTA's counts and rows, and acquires the others'
            last = addAcqRelGpu(p.scr.barrier + 2, 1u) == gridDim.x - 1;
            if (last) p.scr.barrier[2] = p.scr.barrier[3] = 0;
        }
        __syncthreads();
        if (last && fixed) {
            int *counts = reinterpret_cast<int *>(self + p.lay.off_counts);
            for (int e = tid; e < p.E; e += kThreads) {
                const int c = ldVolatile(p.scr.cnt + e);
                if (c > p.rows_per_expert) atomicOr(p.scr.status, ST_CAPACITY);
                counts[e] = c;
                p.recv_count[e] = c;
                p.layout_range[e] = static_cast<unsigned>(c);
                p.expert_offsets[e] = e * p.rows_per_expert;
                if (e == p.E - 1) p.expert_offsets[p.E] = p.E * p.rows_per_expert;
            }
            if (tid == 0) reinterpret_cast<int *>(self + p.lay.off_grp_tokens)[0] = p.topk_weights != nullptr ? p.T : 0;
        }
        if (last && flags_last && (fixed || masked[0] == 0)) {
            // The flags go up behind all counts (of every warp) and, through the exit counter, all rows: a GEMM launched on
            // another stream may look at them while this kernel runs.  It runs on this GPU, the only one of the group, so the
            // release needs no wider scope.
            __syncthreads();
            for (int e = tid; e < p.E; e += kThreads) stReleaseGpu(reinterpret_cast<uint64_t *>(self + p.lay.off_disp_flag) + e, p.epoch);
            if (tid == kThreads - 1) stReleaseGpu(reinterpret_cast<uint64_t *>(self + p.lay.off_counts_flag), p.epoch); // (beside the others, not behind)
        }
        if (last)
            for (int e = tid; e < p.E; e += kThreads) {
                p.scr.cnt[e] = 0;
                p.scr.sent[e] = 0;
            }
    }
}

// ------------------------------------------------------------------ combine

// Logarithmic 10-bit row format for combine (role of the reference's LogFMT-10 codec,
// examples/device/ep/csrc/kernels/nixl_ep_ll.cu:459-616).  The 15-bit magnitude pattern of a bf16
// (exponent and mantissa read as one integer) is a piecewise-linear logarithm of the value, so
// the codec works on patterns with integer and fp32 arithmetic only: per 128-channel group the
// patterns between the smallest non-zero one (at most 32 octaves = 4096 patterns below the
// largest) and the largest are mapped onto 510 steps; code 0 is exact zero and one further bit
// holds the sign.  A group that spans at most 510 patterns (four octaves) is coded exactly;
// otherwise the value is rounded to the nearest grid pattern, a relative error of at most
// (range / 510 + 1) * 2^-8.  Non-finite inputs are clamped to the largest finite bf16.
//
// Layout of a row of H channels (H % 512 == 0) in its H * 2-byte landing slot: H / 512 blocks of
// 160 words; in a block, lane l (16 channels l*16 .. l*16+15 of the block) owns words j*32 + l,
// j < 5, so that a warp's five stores are each one contiguous 128 bytes; words 0..3 and the low
// half of word 4 hold the sixteen 9-bit codes as one little-endian bit stream, the high half of
// word 4 the sixteen sign bits.  After the blocks, at byte H * 10 / 8, one (smallest pattern as
// int32, patterns per step as float) pair per group.
constexpr unsigned kLogFmtSteps = 510;
constexpr int kLogFmtMaxPatterns = 32 * 128;

__device__ __forceinline__ void stPeer4(void *p, uint32_t v) {
    asm volatile("st.global.L1::no_allocate.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ void stPeer8(void *p, const uint2 &v) {
    asm volatile("st.global.L1::no_allocate.v2.u32 [%0], {%1,%2};" ::"l"(p), "r"(v.x), "r"(v.y) : "memory");
}

// Encodes the 16 bf16 values a lane holds; the eight lanes of a 128-channel group cooperate on
// the range.  `meta` is the group's (smallest pattern, patterns per step), identical in the eight lanes.
__device__ __forceinline__ void logfmtEncode16(const uint4 &lo, const uint4 &hi, uint32_t (&w)[5], uint2 &meta) {
    const uint32_t raw[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
    uint32_t pat[16];
    uint32_t signs = 0, pmax = 0, pmin_m1 = 0xffffffffu; // zero patterns wrap to the top and drop out of the minimum
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        signs |= ((raw[i] >> 15) & 1u) << (2 * i);
        signs |= (raw[i] >> 31) << (2 * i + 1);
        pat[2 * i] = min(raw[i] & 0x7fffu, 0x7f7fu);
        pat[2 * i + 1] = min((raw[i] >> 16) & 0x7fffu, 0x7f7fu);
        pmax = max(pmax, max(pat[2 * i], pat[2 * i + 1]));
        pmin_m1 = min(pmin_m1, min(pat[2 * i] - 1u, pat[2 * i + 1] - 1u));
    }
#pragma unroll
    for (int off = 4; off >= 1; off >>= 1) {
        pmax = max(pmax, __shfl_xor_sync(0xffffffffu, pmax, off));
        pmin_m1 = min(pmin_m1, __shfl_xor_sync(0xffffffffu, pmin_m1, off));
    }
    int pmin = pmax ? static_cast<int>(pmin_m1 + 1u) : 0;
    pmin = max(pmin, static_cast<int>(pmax) - kLogFmtMaxPatterns);
    const unsigned range = pmax - static_cast<unsigned>(pmin);
    const bool wide = range > kLogFmtSteps;
    const float scale = wide ? static_cast<float>(kLogFmtSteps) / static_cast<float>(range) : 1.f;
    meta = make_uint2(static_cast<uint32_t>(pmin), __float_as_uint(wide ? static_cast<float>(range) / static_cast<float>(kLogFmtSteps) : 1.f));
    uint64_t acc = 0;
    int bits = 0, wi = 0;
#pragma unroll
    for (int i = 0; i < 16; ++i) {
        const int above = max(static_cast<int>(pat[i]) - pmin, 0);
        const uint32_t code = pat[i] ? 1u + min(__float2uint_rn(static_cast<float>(above) * scale), kLogFmtSteps) : 0u;
        acc |= static_cast<uint64_t>(code) << bits;
        bits += 9;
        if (bits >= 32) {
            w[wi++] = static_cast<uint32_t>(acc);
            acc >>= 32;
            bits -= 32;
        }
    }
    w[4] = static_cast<uint32_t>(acc) | (signs << 16);
}

// acc[i] += weight * value_i for the 16 values of one lane's words.
__device__ __forceinline__ void logfmtDecodeAdd16(const uint32_t (&w)[5], const uint2 &meta, float weight, float (&acc)[16]) {
    const float per_step = __uint_as_float(meta.y);
#pragma unroll
    for (int i = 0; i < 16; ++i) {
        const int bit = 9 * i, idx = bit >> 5, sh = bit & 31;
        const uint32_t next = idx < 4 ? w[idx + 1] : 0u;
        const uint32_t code = __funnelshift_r(w[idx], next, sh) & 0x1ffu;
        const uint32_t pat = meta.x + __float2uint_rn(static_cast<float>(code - 1u) * per_step);
        const uint32_t sign = (w[4] >> (16 + i)) << 31;
        const float v = __uint_as_float(code ? ((pat << 16) | sign) : 0u);
        acc[i] = fmaf(weight, v, acc[i]);
    }
}

// The reduction of pull-mode combine for the tokens of this thread group.  KMAX bounds top-k at
// compile time so that the K rows' 16-byte vectors live in registers.  With kDouble the loads of
// the next vector position are issued before the current one is reduced: a load from a peer takes
// microseconds, and without the overlap every position would pay that latency in full.
template <int KMAX, bool kDouble>
__device__ __forceinline__ void pullReduce(const NixlEpCombineParams &p, int El, int vecs, int nt, int groups_per_cta, int grp, int gtid) {
    __nv_bfloat16 *out = static_cast<__nv_bfloat16 *>(p.out);
    for (int t = blockIdx.x * groups_per_cta + grp; t < p.T; t += gridDim.x * groups_per_cta) {
        float w[KMAX];
        const uint4 *src[KMAX];
#pragma unroll
        for (int k = 0; k < KMAX; ++k) {
            w[k] = __int_as_float(0x7fc00000); // NaN marks "skip" (a real weight may be 0)
            src[k] = nullptr;
            if (k < p.K) {
                const long long e = p.topk_idx[static_cast<long long>(t) * p.K + k];
                const int row = p.send_row[static_cast<long long>(t) * p.K + k];
                if (e >= 0 && e < p.E && row >= 0) {
                    const int r = static_cast<int>(e) / El;
                    char *peer = peerBase(p.peers, r);
                    if (peer != nullptr && ldVolatile(p.scr.mask + r) == 0) {
                        w[k] = p.topk_weights[static_cast<long long>(t) * p.K + k];
                        src[k] = reinterpret_cast<const uint4 *>(peer + p.lay.off_comb_in + static_cast<long long>(row) * p.H * 2);
                    }
                }
            }
        }
        auto load = [&](uint4(&buf)[KMAX], int v) {
#pragma unroll
            for (int k = 0; k < KMAX; ++k)
                if (k < p.K && w[k] == w[k]) buf[k] = ldStream16(src[k] + v);
        };
        auto reduceStore = [&](const uint4(&buf)[KMAX], int v) {
            float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int k = 0; k < KMAX; ++k) {
                if (k >= p.K || w[k] != w[k]) continue;
                const __nv_bfloat162 *h = reinterpret_cast<const __nv_bfloat162 *>(&buf[k]);
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const float2 f = __bfloat1622float2(h[i]);
                    acc[2 * i] = fmaf(w[k], f.x, acc[2 * i]);
                    acc[2 * i + 1] = fmaf(w[k], f.y, acc[2 * i + 1]);
                }
            }
            uint4 o;
            __nv_bfloat162 *oh = reinterpret_cast<__nv_bfloat162 *>(&o);
#pragma unroll
            for (int i = 0; i < 4; ++i) oh[i] = __floats2bfloat162_rn(acc[2 * i], acc[2 * i + 1]);
            *reinterpret_cast<uint4 *>(out + static_cast<long long>(t) * p.H + v * 8) = o;
        };
        if constexpr (kDouble) {
            uint4 a[KMAX], b[KMAX];
            int v = gtid;
            if (v < vecs) load(a, v);
            while (v < vecs) {
                const int v1 = v + nt;
                if (v1 < vecs) load(b, v1);
                reduceStore(a, v);
                if (v1 >= vecs) break;
                const int v2 = v1 + nt;
                if (v2 < vecs) load(a, v2);
                reduceStore(b, v1);
                v = v2;
            }
        } else {
            for (int v = gtid; v < vecs; v += nt) {
                uint4 raw[KMAX];
                load(raw, v);
                reduceStore(raw, v);
            }
        }
    }
}

// Pull-mode combine: announce that this rank's expert outputs are complete, wait for the same
// word from every peer, then each token's home rank loads the K rows from where dispatch put
// them and reduces in fp32.  Every row crosses NVLink once and is never staged.
__device__ __forceinline__ void epCombinePull(const NixlEpCombineParams &p) {
    const int El = p.E / p.R;
    const int tid = threadIdx.x;
    char *self = peerBase(p.peers, p.rank);
    const int vecs = p.H / 8;
    if ((p.phases & 1) && blockIdx.x == 0 && tid < p.R) {
        char *peer = peerBase(p.peers, tid);
        if (peer != nullptr && ldVolatile(p.scr.mask + tid) == 0) {
            __threadfence_system();
            stReleaseSys(reinterpret_cast<uint64_t *>(peer + p.lay.off_comb_flag) + p.rank, p.epoch);
        }
    }
    if (!(p.phases & 2)) return;
    const uint64_t *flag = reinterpret_cast<const uint64_t *>(self + p.lay.off_comb_flag);
    if (tid < p.R && ldVolatile(p.scr.mask + tid) == 0 && peerBase(p.peers, tid) != nullptr) {
        if (!waitFlag(flag + tid, p.epoch, p.timeout_ns)) {
            atomicExch(p.scr.mask + tid, 1);
            atomicOr(p.scr.status, ST_PEER_TIMEOUT);
        }
    }
    __syncthreads();
    const int nt = threadsPerItem(p.T);
    const int groups_per_cta = kThreads / nt;
    const int grp = tid / nt, gtid = tid - grp * nt;
    if (p.K <= 8) pullReduce<8, true>(p, El, vecs, nt, groups_per_cta, grp, gtid);
    else pullReduce<kMaxTopk, false>(p, El, vecs, nt, groups_per_cta, grp, gtid);
}

// Staging area of one warp of the rank-reduced combine: kRrSlots 16-byte slots per lane, filled by asynchronous
// copies.  Loads that wait in shared memory instead of registers let a warp keep 12 KB in flight, and two CTAs fit
// on an SM.
constexpr int kRrSlots = 24;
constexpr int kRrWarpBytes = kRrSlots * 32 * 16;
constexpr int kRrCtaBytes = (kThreads / 32) * kRrWarpBytes;

__device__ __forceinline__ void cpAsync16(uint32_t smem_addr, const void *g) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_addr), "l"(g) : "memory"); // through L2: sees what peers wrote
}
__device__ __forceinline__ void cpAsyncWaitAll() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// One warp: dst[v] = sum over the n rows (1..8) of w[k] * src[k][v] for the row's `vecs` 16-byte vectors, fp32
// accumulation, bf16 out.  kRrSlots / n vector positions of every row are in flight per lane.  Each lane reads back
// only the slots it filled itself, so its own wait is all the synchronisation the area needs.  dst may be a peer's memory.
__device__ __forceinline__ void warpWeightedRows(int n, const uint4 *const (&src)[8], const float (&w)[8], uint4 *dst, int vecs, int lane,
                                                 uint4 *stage) {
    const int per_pass = kRrSlots / n;
    const uint32_t sbase = static_cast<uint32_t>(__cvta_generic_to_shared(stage)) + lane * 16;
    for (int v0 = lane; v0 < vecs; v0 += 32 * per_pass) {
#pragma unroll 1
        for (int u = 0; u < per_pass; ++u) {
            const int v = v0 + u * 32;
            if (v >= vecs) break;
#pragma unroll
            for (int k = 0; k < 8; ++k)
                if (k < n) cpAsync16(sbase + static_cast<uint32_t>((u * n + k) * 32 * 16), src[k] + v);
        }
        cpAsyncWaitAll();
#pragma unroll 1
        for (int u = 0; u < per_pass; ++u) {
            const int v = v0 + u * 32;
            if (v >= vecs) break;
            float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                if (k >= n) continue;
                const uint4 raw = stage[(u * n + k) * 32 + lane];
                const __nv_bfloat162 *h = reinterpret_cast<const __nv_bfloat162 *>(&raw);
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const float2 f = __bfloat1622float2(h[j]);
                    acc[2 * j] = fmaf(w[k], f.x, acc[2 * j]);
                    acc[2 * j + 1] = fmaf(w[k], f.y, acc[2 * j + 1]);
                }
            }
            uint4 o;
            __nv_bfloat162 *oh = reinterpret_cast<__nv_bfloat162 *>(&o);
#pragma unroll
            for (int j = 0; j < 4; ++j) oh[j] = __floats2bfloat162_rn(acc[2 * j], acc[2 * j + 1]);
            stPeer16(dst + v, o);
        }
    }
}

// Rank-reduced combine (NixlEpCombineParams::max_tokens).  Phase 1, expert rank: one warp per (token, home
// rank) group record adds the token's rows up in fp32, weighted, and stores ONE bf16 row at the home rank.
// Phase 2, home rank: add the rows of the ranks the token went to.
template <int kPhases>
__device__ __forceinline__ void epCombineRankReduce(const NixlEpCombineParams &p) {
    const int El = p.E / p.R;
    const int tid = threadIdx.x, lane = tid & 31;
    char *self = peerBase(p.peers, p.rank);
    const int vecs = p.H / 8;
    const long long M = p.max_tokens;
    const int tag = static_cast<int>(p.epoch & 0x7fffffffull);
    extern __shared__ __align__(16) unsigned char rr_stage[];
    uint4 *stage = reinterpret_cast<uint4 *>(rr_stage + (tid >> 5) * kRrWarpBytes);

    if constexpr ((kPhases & 1) != 0) {
        const __nv_bfloat16 *x = static_cast<const __nv_bfloat16 *>(p.x);
        const int *tokens_of = reinterpret_cast<const int *>(self + p.lay.off_grp_tokens);
        const uint4 *records = reinterpret_cast<const uint4 *>(self + p.lay.off_grp);
        int max_t = 0;
        for (int r = 0; r < p.R; ++r) {
            const int n = ldVolatile(tokens_of + r);
            max_t = n > max_t ? (n < M ? n : static_cast<int>(M)) : max_t;
        }
        const long long items = static_cast<long long>(max_t) * p.R;
        const long long warps = static_cast<long long>(gridDim.x) * (kThreads / 32);
        // item = token * R + home rank: neighbouring warps store to different peers
        for (long long i = static_cast<long long>(blockIdx.x) * (kThreads / 32) + (tid >> 5); i < items; i += warps) {
            const int r = static_cast<int>(i % p.R);
            const long long t = i / p.R;
            if (t >= ldVolatile(tokens_of + r) || ldVolatile(p.scr.mask + r) != 0) continue;
            char *peer = peerBase(p.peers, r);
            if (peer == nullptr) continue;
            const uint4 *rec = records + (static_cast<long long>(r) * M + t) * 5;
            const uint4 head = rec[0];
            const int n = static_cast<int>(head.x);
            if (static_cast<int>(head.y) != tag || n <= 0 || n > 8) continue;
            const uint4 r0 = rec[1], r1 = rec[2], w0 = rec[3], w1 = rec[4];
            const int rows[8] = {int(r0.x), int(r0.y), int(r0.z), int(r0.w), int(r1.x), int(r1.y), int(r1.z), int(r1.w)};
            const float w[8] = {__uint_as_float(w0.x), __uint_as_float(w0.y), __uint_as_float(w0.z), __uint_as_float(w0.w),
                                __uint_as_float(w1.x), __uint_as_float(w1.y), __uint_as_float(w1.z), __uint_as_float(w1.w)};
            const uint4 *src[8];
            float wk[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                src[k] = reinterpret_cast<const uint4 *>(x + static_cast<long long>(k < n ? rows[k] : rows[0]) * p.H);
                wk[k] = k < n ? w[k] : 0.f; // padding rows repeat the first one with weight zero
            }
            uint4 *dst = reinterpret_cast<uint4 *>(peer + p.lay.off_comb_x + (static_cast<long long>(p.rank) * M + t) * p.H * 2);
            warpWeightedRows(n, src, wk, dst, vecs, lane, stage);
        }
        __syncthreads();
        if (tid == 0) __threadfence_system();
        gridBarrier(p.scr.barrier, p.scr.status, p.timeout_ns);
        // Everybody's rows are out: tell each home rank.
        for (int d = blockIdx.x; d < p.R; d += gridDim.x) {
            if (ldVolatile(p.scr.mask + d) != 0) continue;
            char *peer = peerBase(p.peers, d);
            if (peer != nullptr && tid == 0) {
                __threadfence_system();
                stReleaseSys(reinterpret_cast<uint64_t *>(peer + p.lay.off_comb_flag) + p.rank, p.epoch);
            }
        }
    }

    if constexpr ((kPhases & 2) != 0) {
        const uint64_t *flag = reinterpret_cast<const uint64_t *>(self + p.lay.off_comb_flag);
        if (tid < p.R && ldVolatile(p.scr.mask + tid) == 0 && peerBase(p.peers, tid) != nullptr) {
            if (!waitFlag(flag + tid, p.epoch, p.timeout_ns)) {
                atomicExch(p.scr.mask + tid, 1);
                atomicOr(p.scr.status, ST_PEER_TIMEOUT);
            }
        }
        __syncthreads();
        const __nv_bfloat16 *landing = reinterpret_cast<const __nv_bfloat16 *>(self + p.lay.off_comb_x);
        __nv_bfloat16 *out = static_cast<__nv_bfloat16 *>(p.out);
        const int warps = gridDim.x * (kThreads / 32);
        for (int t = blockIdx.x * (kThreads / 32) + (tid >> 5); t < p.T; t += warps) { // one warp per token
            // ranks that hold copies of this token (and answered)
            unsigned ranks = 0;
            for (int k = 0; k < p.K; ++k) {
                const long long e = p.topk_idx[static_cast<long long>(t) * p.K + k];
                if (e >= 0 && e < p.E && ldVolatile(p.scr.mask + static_cast<int>(e) / El) == 0) ranks |= 1u << (static_cast<int>(e) / El);
            }
            uint4 *dst = reinterpret_cast<uint4 *>(out + static_cast<long long>(t) * p.H);
            if (ranks == 0) {
                for (int v = lane; v < vecs; v += 32) dst[v] = make_uint4(0u, 0u, 0u, 0u);
                continue;
            }
            if (__popc(ranks) <= 8) {
                const uint4 *src[8];
                float one[8];
                unsigned left = ranks;
                const int first = __ffs(ranks) - 1;
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const int d = left ? __ffs(left) - 1 : first;
                    one[j] = left ? 1.f : 0.f;
                    left &= left - 1; // (0 stays 0)
                    src[j] = reinterpret_cast<const uint4 *>(landing + (static_cast<long long>(d) * M + t) * p.H);
                }
                warpWeightedRows(__popc(ranks), src, one, dst, vecs, lane, stage);
                continue;
            }
            for (int v = lane; v < vecs; v += 32) { // more than eight ranks hold copies: plain loads, eight rows at a time
                float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
                unsigned left = ranks;
                while (left) {
                    const int d = __ffs(left) - 1;
                    left &= left - 1;
                    const uint4 raw = *reinterpret_cast<const uint4 *>(landing + (static_cast<long long>(d) * M + t) * p.H + v * 8);
                    const __nv_bfloat162 *h = reinterpret_cast<const __nv_bfloat162 *>(&raw);
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const float2 f = __bfloat1622float2(h[i]);
                        acc[2 * i] += f.x;
                        acc[2 * i + 1] += f.y;
                    }
                }
                uint4 o;
                __nv_bfloat162 *oh = reinterpret_cast<__nv_bfloat162 *>(&o);
#pragma unroll
                for (int i = 0; i < 4; ++i) oh[i] = __floats2bfloat162_rn(acc[2 * i], acc[2 * i + 1]);
                dst[v] = o;
            }
        }
    }
}

// The rank-reduced mode as two kernels of its own: each phase alone needs few enough registers for two CTAs per SM,
// which is what keeps enough loads in flight; the second launch starts when every CTA of the first has left.
__global__ void __launch_bounds__(kThreads, 2) epCombineRankReduceSend(const __grid_constant__ NixlEpCombineParams p) { epCombineRankReduce<1>(p); }
__global__ void __launch_bounds__(kThreads, 2) epCombineRankReduceRecv(const __grid_constant__ NixlEpCombineParams p) { epCombineRankReduce<2>(p); }

__global__ void __launch_bounds__(kThreads) epCombineKernel(const __grid_constant__ NixlEpCombineParams p) {
    __shared__ int offs[kMaxRanks * 8 + 1]; // expert_offsets copy (El + 1 <= 513)
    __shared__ int cnts[kMaxRanks * 8];
    const int El = p.E / p.R;
    const int tid = threadIdx.x;
    char *self = peerBase(p.peers, p.rank);
    const int vecs = p.H / 8;

    if (p.pull) {
        epCombinePull(p);
        return;
    }

    if (p.phases & 1) {
        for (int i = tid; i <= El; i += kThreads) offs[i] = p.expert_offsets[i];
        for (int i = tid; i < El; i += kThreads) cnts[i] = p.recv_count[i];
        __syncthreads();
        // Rows are enumerated expert by expert; every warp of the grid takes every n-th valid row.
        const __nv_bfloat16 *x = static_cast<const __nv_bfloat16 *>(p.x);
        const int lane = tid & 31;
        const long long warps = static_cast<long long>(gridDim.x) * (kThreads / 32);
        int le = 0, seen = 0; // rows of experts < le
        for (long long j = static_cast<long long>(blockIdx.x) * (kThreads / 32) + (tid >> 5);; j += warps) {
            while (le < El && j >= seen + cnts[le]) seen += cnts[le++];
            if (le >= El) break;
            const long long row = static_cast<long long>(offs[le]) + (j - seen);
            const uint2 info = *reinterpret_cast<const uint2 *>(p.recv_info + row * 2);
            const int r = static_cast<int>(info.x);
            if (r < 0 || r >= p.R || ldVolatile(p.scr.mask + r) != 0) continue;
            char *peer = peerBase(p.peers, r);
            if (peer == nullptr) continue;
            const uint4 *src = reinterpret_cast<const uint4 *>(x + row * p.H);
            uint4 *dst = reinterpret_cast<uint4 *>(peer + p.lay.off_comb_x + static_cast<long long>(info.y) * p.H * 2);
            if (p.use_logfmt) {
                uint32_t *words = reinterpret_cast<uint32_t *>(dst);
                uint2 *meta = reinterpret_cast<uint2 *>(reinterpret_cast<char *>(dst) + static_cast<long long>(p.H) * 10 / 8);
                const int blocks = p.H / 512;
                uint4 lo = ldStream16(src + lane * 2), hi = ldStream16(src + lane * 2 + 1);
                for (int b = 0; b < blocks; ++b) {
                    uint4 nlo = lo, nhi = hi;
                    if (b + 1 < blocks) { // next block's loads fly while this one is encoded
                        nlo = ldStream16(src + (b + 1) * 64 + lane * 2);
                        nhi = ldStream16(src + (b + 1) * 64 + lane * 2 + 1);
                    }
                    uint32_t w[5];
                    uint2 m;
                    logfmtEncode16(lo, hi, w, m);
#pragma unroll
                    for (int j = 0; j < 5; ++j) stPeer4(words + b * 160 + j * 32 + lane, w[j]);
                    if ((lane & 7) == 0) stPeer8(meta + b * 4 + (lane >> 3), m);
                    lo = nlo;
                    hi = nhi;
                }
                continue;
            }
            for (int v0 = lane; v0 < vecs; v0 += 8 * 32) { // eight loads in flight per lane
                uint4 val[8];
#pragma unroll
                for (int i = 0; i < 8; ++i)
                    if (v0 + i * 32 < vecs) val[i] = ldStream16(src + v0 + i * 32);
#pragma unroll
                for (int i = 0; i < 8; ++i)
                    if (v0 + i * 32 < vecs) stPeer16(dst + v0 + i * 32, val[i]);
            }
        }
        __syncthreads();
        if (tid == 0) __threadfence_system();
        gridBarrier(p.scr.barrier, p.scr.status, p.timeout_ns);
        // Everybody's rows are out: tell each source rank.
        for (int d = blockIdx.x; d < p.R; d += gridDim.x) {
            if (ldVolatile(p.scr.mask + d) != 0) continue;
            char *peer = peerBase(p.peers, d);
            if (peer != nullptr && tid == 0) {
                __threadfence_system();
                stReleaseSys(reinterpret_cast<uint64_t *>(peer + p.lay.off_comb_flag) + p.rank, p.epoch);
            }
        }
    }

    if (p.phases & 2) {
        const uint64_t *flag = reinterpret_cast<const uint64_t *>(self + p.lay.off_comb_flag);
        if (tid < p.R && ldVolatile(p.scr.mask + tid) == 0 && peerBase(p.peers, tid) != nullptr) {
            if (!waitFlag(flag + tid, p.epoch, p.timeout_ns)) {
                atomicExch(p.scr.mask + tid, 1);
                atomicOr(p.scr.status, ST_PEER_TIMEOUT);
            }
        }
        __syncthreads();
        // out[t] = sum_k w[t,k] * y[t,k] in fp32
        const __nv_bfloat16 *landing = reinterpret_cast<const __nv_bfloat16 *>(self + p.lay.off_comb_x);
        __nv_bfloat16 *out = static_cast<__nv_bfloat16 *>(p.out);
        const int nt = threadsPerItem(p.T);
        const int groups_per_cta = kThreads / nt;
        const int grp = tid / nt, gtid = tid - grp * nt;
        for (int t = blockIdx.x * groups_per_cta + grp; t < p.T; t += gridDim.x * groups_per_cta) {
            float w[kMaxTopk];
#pragma unroll
            for (int k = 0; k < kMaxTopk; ++k) {
                w[k] = 0.f;
                if (k < p.K) {
                    const long long e = p.topk_idx[static_cast<long long>(t) * p.K + k];
                    if (e >= 0 && e < p.E && ldVolatile(p.scr.mask + static_cast<int>(e) / El) == 0)
                        w[k] = p.topk_weights[static_cast<long long>(t) * p.K + k];
                    else w[k] = __int_as_float(0x7fc00000); // NaN marks "skip" (a real weight may be 0)
                }
            }
            if (p.use_logfmt) {
                const long long meta_off = static_cast<long long>(p.H) * 10 / 8;
                for (int u = gtid; u < p.H / 16; u += nt) {
                    const int b = u >> 5, l = u & 31;
                    float acc[16];
#pragma unroll
                    for (int i = 0; i < 16; ++i) acc[i] = 0.f;
#pragma unroll
                    for (int k0 = 0; k0 < kMaxTopk; k0 += 4) { // four rows' words in flight
                        if (k0 >= p.K) break;
                        uint32_t cw[4][5];
                        uint2 m[4];
#pragma unroll
                        for (int kk = 0; kk < 4; ++kk) {
                            const int k = k0 + kk;
                            if (k < p.K && w[k] == w[k]) {
                                const char *slot = reinterpret_cast<const char *>(landing + (static_cast<long long>(t) * p.K + k) * p.H);
                                const uint32_t *words = reinterpret_cast<const uint32_t *>(slot) + b * 160 + l;
#pragma unroll
                                for (int j = 0; j < 5; ++j) cw[kk][j] = words[j * 32];
                                m[kk] = *reinterpret_cast<const uint2 *>(slot + meta_off + (b * 4 + (l >> 3)) * 8);
                            }
                        }
#pragma unroll
                        for (int kk = 0; kk < 4; ++kk) {
                            const int k = k0 + kk;
                            if (k < p.K && w[k] == w[k]) logfmtDecodeAdd16(cw[kk], m[kk], w[k], acc);
                        }
                    }
                    uint4 o[2];
                    __nv_bfloat162 *oh = reinterpret_cast<__nv_bfloat162 *>(o);
#pragma unroll
                    for (int i = 0; i < 8; ++i) oh[i] = __floats2bfloat162_rn(acc[2 * i], acc[2 * i + 1]);
                    uint4 *dst = reinterpret_cast<uint4 *>(out + static_cast<long long>(t) * p.H + b * 512 + l * 16);
                    dst[0] = o[0];
                    dst[1] = o[1];
                }
                continue;
            }
            for (int v = gtid; v < vecs; v += nt) {
                float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
                uint4 raw[kMaxTopk];
#pragma unroll
                for (int k = 0; k < kMaxTopk; ++k)
                    if (k < p.K && w[k] == w[k])
                        raw[k] = *reinterpret_cast<const uint4 *>(landing + (static_cast<long long>(t) * p.K + k) * p.H + v * 8);
#pragma unroll
                for (int k = 0; k < kMaxTopk; ++k) {
                    if (k >= p.K || w[k] != w[k]) continue;
                    const __nv_bfloat162 *h = reinterpret_cast<const __nv_bfloat162 *>(&raw[k]);
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const float2 f = __bfloat1622float2(h[i]);
                        acc[2 * i] = fmaf(w[k], f.x, acc[2 * i]);
                        acc[2 * i + 1] = fmaf(w[k], f.y, acc[2 * i + 1]);
                    }
                }
                uint4 o;
                __nv_bfloat162 *oh = reinterpret_cast<__nv_bfloat162 *>(&o);
#pragma unroll
                for (int i = 0; i < 4; ++i) oh[i] = __floats2bfloat162_rn(acc[2 * i], acc[2 * i + 1]);
                *reinterpret_cast<uint4 *>(out + static_cast<long long>(t) * p.H + v * 8) = o;
            }
        }
    }
}

// Combine when one rank holds every expert (R == 1): nothing has to travel, so whatever the mode the result is the weighted
// sum of the token's rows of x where they lie.  One kernel without flags, barriers or a landing zone, for calls that send and
// receive in one launch into an output apart from x (nixl_ep_combine_launch).  A warp takes a token or a part of one.  Bound by memory (K rows read,
// one written), measured on one B200, 32 experts, top-8: 4096 tokens x 7168 83 us (528 MB, 6.4 TB/s), where the two kernels of
// the rank-reduced mode took 107 + 34 us; 128 tokens, low-latency layout 4.9 us, where the push mode's copy to the landing zone,
// barrier and sum took 27.6 us.
template <int NR>
__device__ __forceinline__ void localRows(int n, const uint4 *const (&src)[NR], const float (&w)[NR], uint4 *dst, int vecs, int v0, int step) {
    for (int v = v0; v < vecs; v += step) {
        uint4 raw[NR];
#pragma unroll
        for (int k = 0; k < NR; ++k) {
            raw[k] = make_uint4(0u, 0u, 0u, 0u);
            if (k < n) raw[k] = ldStream16(src[k] + v);
        }
        float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int k = 0; k < NR; ++k) {
            if (k >= n) continue;
            const __nv_bfloat162 *h = reinterpret_cast<const __nv_bfloat162 *>(&raw[k]);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float2 f = __bfloat1622float2(h[j]);
                acc[2 * j] = fmaf(w[k], f.x, acc[2 * j]);
                acc[2 * j + 1] = fmaf(w[k], f.y, acc[2 * j + 1]);
            }
        }
        uint4 o;
        __nv_bfloat162 *oh = reinterpret_cast<__nv_bfloat162 *>(&o);
#pragma unroll
        for (int j = 0; j < 4; ++j) oh[j] = __floats2bfloat162_rn(acc[2 * j], acc[2 * j + 1]);
        stPeer16(dst + v, o);
    }
}

// The same for rows in the logarithmic format: each row is coded and decoded in registers, as it would be on its way out
// and in, so the result is what the coded path gives.  Slices of 512 channels, 16 per lane.
template <int NR>
__device__ __forceinline__ void localRowsCoded(int n, const uint4 *const (&src)[NR], const float (&w)[NR], uint4 *dst, int slices, int first, int step, int lane) {
    for (int b = first; b < slices; b += step) {
        float acc[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) acc[i] = 0.f;
        const int at = b * 64 + lane * 2;
        uint4 lo = ldStream16(src[0] + at), hi = ldStream16(src[0] + at + 1);
#pragma unroll
        for (int k = 0; k < NR; ++k) {
            if (k >= n) break;
            uint4 nlo = lo, nhi = hi;
            if (k + 1 < NR && k + 1 < n) { // the next row's loads fly while this one is coded
                nlo = ldStream16(src[k + 1 < NR ? k + 1 : k] + at);
                nhi = ldStream16(src[k + 1 < NR ? k + 1 : k] + at + 1);
            }
            uint32_t code[5];
            uint2 meta;
            logfmtEncode16(lo, hi, code, meta);
            logfmtDecodeAdd16(code, meta, w[k], acc);
            lo = nlo;
            hi = nhi;
        }
        uint4 o[2];
        __nv_bfloat162 *oh = reinterpret_cast<__nv_bfloat162 *>(o);
#pragma unroll
        for (int i = 0; i < 8; ++i) oh[i] = __floats2bfloat162_rn(acc[2 * i], acc[2 * i + 1]);
        stPeer16(dst + at, o[0]);
        stPeer16(dst + at + 1, o[1]);
    }
}

template <int NR, bool kCoded>
__global__ void __launch_bounds__(kThreads, NR <= 8 && !kCoded ? 3 : 2) epCombineLocal(const __grid_constant__ NixlEpCombineParams p, int parts) {
    nixl_pdl::allowNextKernel();
    nixl_pdl::waitForPreviousKernel();
    const int lane = threadIdx.x & 31;
    const int vecs = p.H / 8;
    const char *self = peerBase(p.peers, p.rank);
    const bool off = ldVolatile(p.scr.mask) != 0;
    const __nv_bfloat16 *x = static_cast<const __nv_bfloat16 *>(p.x);
    const long long items = static_cast<long long>(p.T) * parts;
    // consecutive parts and tokens on different SMs
    for (long long i = static_cast<long long>(threadIdx.x >> 5) * gridDim.x + blockIdx.x; i < items; i += static_cast<long long>(gridDim.x) * (kThreads / 32)) {
        const long long t = i / parts;
        const int part = static_cast<int>(i - t * parts);
        // Lane k: row and weight of one copy, -1 when there is none.
        int row = -1;
        float weight = 0.f;
        if (p.pull == 2) { // rank-reduced mode: rows and weights as the dispatch recorded them, for tokens that still have an expert
            const NixlEpGroupRecord *rec = reinterpret_cast<const NixlEpGroupRecord *>(self + p.lay.off_grp) + t;
            const long long e = lane < p.K ? p.topk_idx[t * p.K + lane] : -1;
            if (lane < 8 && !off && rec->pad[0] == static_cast<int>(p.epoch & 0x7fffffffull) && lane < rec->n) {
                row = rec->rows[lane];
                weight = rec->w[lane];
            }
            if (!__any_sync(0xffffffffu, e >= 0 && e < p.E)) row = -1; // (looked at last: its load is in flight beside the record's)
        } else if (lane < p.K) {
            const long long e = p.topk_idx[t * p.K + lane];
            if (e >= 0 && e < p.E && !off) row = p.send_row[t * p.K + lane];
            weight = p.topk_weights[t * p.K + lane];
            if (weight != weight) row = -1; // a NaN weight drops the copy
        }
        const unsigned have = __ballot_sync(0xffffffffu, row >= 0);
        const int n = __popc(have);
        const uint4 *src[NR];
        float w[NR];
        unsigned left = have;
#pragma unroll
        for (int k = 0; k < NR; ++k) { // in the copies' order
            const int from = left ? __ffs(left) - 1 : 0;
            left &= left - 1;
            src[k] = reinterpret_cast<const uint4 *>(x + static_cast<long long>(__shfl_sync(0xffffffffu, row, from)) * p.H);
            w[k] = __shfl_sync(0xffffffffu, weight, from);
        }
        uint4 *dst = reinterpret_cast<uint4 *>(static_cast<__nv_bfloat16 *>(p.out) + t * p.H);
        if (!kCoded || n == 0) localRows<NR>(n, src, w, dst, vecs, part * 32 + lane, 32 * parts);
        else localRowsCoded<NR>(n, src, w, dst, p.H / 512, part, parts, lane);
    }
}

// ------------------------------------------------------------------ dispatch layout (counts only)

// Per-rank and per-expert token counts and the token x rank membership matrix of a routing table
// (what the reference computes in examples/device/ep/csrc/kernels/layout.cu before a
// high-throughput dispatch).  Dispatch here does its own counting; this kernel serves callers that
// want the numbers up front (capacity planning, load-balance statistics).
__global__ void __launch_bounds__(256) epLayoutKernel(const int64_t *topk_idx, int T, int K, int E, int R, int *per_rank, int *per_expert,
                                                      unsigned char *in_rank) {
    extern __shared__ int hist[]; // [E] experts, then [R] ranks
    int *h_expert = hist, *h_rank = hist + E;
    for (int i = threadIdx.x; i < E + R; i += blockDim.x) hist[i] = 0;
    __syncthreads();
    const int El = E / R;
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < T; t += gridDim.x * blockDim.x) {
        unsigned long long mask = 0;
        for (int k = 0; k < K; ++k) {
            const long long e = topk_idx[static_cast<long long>(t) * K + k];
            if (e < 0 || e >= E) continue;
            atomicAdd(h_expert + e, 1);
            mask |= 1ull << (static_cast<int>(e) / El);
        }
        for (int r = 0; r < R; ++r) {
            const bool in = (mask >> r) & 1ull;
            in_rank[static_cast<long long>(t) * R + r] = in ? 1 : 0;
            if (in) atomicAdd(h_rank + r, 1);
        }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < E; i += blockDim.x)
        if (h_expert[i]) atomicAdd(per_expert + i, h_expert[i]);
    for (int i = threadIdx.x; i < R; i += blockDim.x)
        if (h_rank[i]) atomicAdd(per_rank + i, h_rank[i]);
}

// ------------------------------------------------------------------ barrier across ranks

__global__ void epBarrierKernel(const void *peers, int64_t off_flags, int R, int rank, uint64_t epoch, uint64_t timeout_ns, int *status,
                                int *mask) {
    const int r = threadIdx.x;
    if (r >= R) return;
    char *peer = peerBase(peers, r);
    if (peer == nullptr || ldVolatile(mask + r) != 0) return;
    __threadfence_system();
    stReleaseSys(reinterpret_cast<uint64_t *>(peer + off_flags) + rank, epoch);
    const uint64_t *mine = reinterpret_cast<const uint64_t *>(peerBase(peers, rank) + off_flags);
    if (!waitFlag(mine + r, epoch, timeout_ns)) {
        atomicExch(mask + r, 1);
        atomicOr(status, ST_PEER_TIMEOUT);
    }
}

int coopGrid(const void *kernel, int requested, size_t smem) {
    int dev = 0, sms = 0, per_sm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kThreads, smem);
    const int limit = sms * (per_sm > 0 ? per_sm : 1);
    int grid = requested > 0 ? requested : sms;
    return grid > limit ? limit : grid;
}

} // namespace

extern "C" int nixl_ep_dispatch_launch(const NixlEpDispatchParams *params, void *stream) {
    if (!params || !params->peers || !params->topk_idx || (!params->x && (params->phases & 1))) return cudaErrorInvalidValue;
    const NixlEpDispatchParams &p = *params;
    if (p.R <= 0 || p.R > kMaxRanks || p.E <= 0 || p.E % p.R || p.K <= 0 || p.K > kMaxTopk || p.H <= 0 || p.H % kGroup ||
        p.E / p.R > kMaxRanks * 8 || p.rank < 0 || p.rank >= p.R || p.T < 0)
        return cudaErrorInvalidValue;
    if (p.H % 512) return cudaErrorInvalidValue; // whole warps per pass; scales move as float4
    if (p.topk_weights && (p.K > 8 || p.R > 32 || p.max_tokens < p.T)) return cudaErrorInvalidValue; // a group record holds eight copies
    if (p.rows_per_expert > 0 && static_cast<long long>(p.rows_per_expert) < static_cast<long long>(p.R) * p.T) return cudaErrorInvalidValue;
    const int tables = dispatchTables(p.E, p.K);
    const size_t smem = dispatchSmem(p.E, p.K, tables);
    const void *kernel = tables == 3 ? reinterpret_cast<const void *>(epDispatchKernel<true>) : reinterpret_cast<const void *>(epDispatchKernel<false>);
    if (smem > 48 * 1024) { // many experts: the shared-memory limit is a per-device function attribute, raised once to all there is
        static bool attr_done[64] = {};
        int dev = 0;
        cudaGetDevice(&dev);
        if (dev < 0 || dev >= 64 || !attr_done[dev]) {
            cudaError_t e = cudaFuncSetAttribute(epDispatchKernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kDispatchSmemMax));
            if (e == cudaSuccess) e = cudaFuncSetAttribute(epDispatchKernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kDispatchSmemMax));
            if (e != cudaSuccess) return e;
            if (dev >= 0 && dev < 64) attr_done[dev] = true;
        }
    }
    // With many tokens four CTAs per SM keep enough loads and stores in flight; a few tokens go to one CTA per SM, whose
    // eight warps share them (fewer CTAs at the grid barrier).
    int requested = p.grid;
    if (requested <= 0) {
        int dev = 0, sms = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        // (CTAs without a token would only add to the barrier and the exit count; the ranks' counts are spread over CTAs.)
        if (p.T >= 4 * sms) requested = kDispatchCtas * sms;
        else if (p.T < sms) requested = p.T > p.R ? p.T : p.R;
    }
    const int grid = coopGrid(kernel, requested, smem);
    void *args[] = {const_cast<NixlEpDispatchParams *>(params)};
    if (placesAreFixed(p)) // no CTA waits for another
        return nixl_pdl::launch(tables == 3 ? epDispatchKernel<true> : epDispatchKernel<false>, grid, kThreads, smem, static_cast<cudaStream_t>(stream), p);
    return cudaLaunchCooperativeKernel(kernel, dim3(grid), dim3(kThreads), args, smem, static_cast<cudaStream_t>(stream));
}

extern "C" int nixl_ep_combine_launch(const NixlEpCombineParams *params, void *stream) {
    if (!params || !params->peers || !params->topk_idx) return cudaErrorInvalidValue;
    const NixlEpCombineParams &p = *params;
    if (p.pull == 1 && !p.send_row) return cudaErrorInvalidValue;
    if (p.pull == 2 && (p.max_tokens <= 0 || p.R > 32 || p.T > p.max_tokens || !p.x)) return cudaErrorInvalidValue;
    if (p.use_logfmt && (p.pull || p.H % 512)) return cudaErrorInvalidValue;
    if (p.R <= 0 || p.R > kMaxRanks || p.E <= 0 || p.E % p.R || p.K <= 0 || p.K > kMaxTopk || p.H <= 0 || p.H % 8 ||
        p.E / p.R > kMaxRanks * 8 || p.rank < 0 || p.rank >= p.R)
        return cudaErrorInvalidValue;
    void *args[] = {const_cast<NixlEpCombineParams *>(params)};
    // A one-rank group sums its rows where they lie, in one pass that writes out while it still reads x: only when both phases
    // are one launch (a send alone must leave out untouched and x free to be overwritten) and out does not overlap x (the
    // other paths have read all of x before the first row of out is written).
    const uintptr_t x0 = reinterpret_cast<uintptr_t>(p.x), out0 = reinterpret_cast<uintptr_t>(p.out);
    const uintptr_t x_bytes = p.x_rows > 0 ? static_cast<uintptr_t>(p.x_rows) * p.H * 2 : 0, out_bytes = static_cast<uintptr_t>(p.T > 0 ? p.T : 0) * p.H * 2;
    const bool apart = x_bytes > 0 && (out0 + out_bytes <= x0 || x0 + x_bytes <= out0);
    if (p.R == 1 && (p.phases & 3) == 3 && apart && p.x && p.topk_weights && p.out && (p.pull == 2 || p.send_row)) {
        if (p.T <= 0) return cudaSuccess;
        int dev = 0, sms = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        // Three CTAs per SM; parts so that every warp has about four items, or as many as a token has slices (512 bytes; coded
        // rows 512 channels, whose coding is a long chain of arithmetic per warp).
        const int ctas = p.grid > 0 ? (p.pull == 2 ? 2 : 1) * p.grid : 3 * sms;
        const long long items = 4LL * ctas * (kThreads / 32);
        const int most = p.use_logfmt ? p.H / 512 : p.H / 256;
        int parts = static_cast<int>(items / p.T < 16 ? items / p.T : 16);
        parts = parts < 1 ? 1 : parts > most ? (most > 0 ? most : 1) : parts;
        const long long want = static_cast<long long>(p.T) * parts;
        const int grid = static_cast<int>(want < ctas ? want : ctas);
        const auto kernel = p.K <= 8 ? (p.use_logfmt ? epCombineLocal<8, true> : epCombineLocal<8, false>)
                                     : (p.use_logfmt ? epCombineLocal<kMaxTopk, true> : epCombineLocal<kMaxTopk, false>);
        static std::atomic<bool> l1_done[4][64];
        if (const cudaError_t e = nixl_pdl::preferL1(reinterpret_cast<const void *>(kernel), dev, l1_done[(p.K <= 8) * 2 + (p.use_logfmt != 0)]); e != cudaSuccess) return e;
        return nixl_pdl::launch(kernel, grid, kThreads, 0, static_cast<cudaStream_t>(stream), p, parts);
    }
    if (p.pull == 2) {
        int dev = 0, sms = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        static bool attr_done[64] = {};
        if (dev >= 0 && dev < 64 && !attr_done[dev]) {
            cudaError_t e = cudaFuncSetAttribute(epCombineRankReduceSend, cudaFuncAttributeMaxDynamicSharedMemorySize, kRrCtaBytes);
            if (e == cudaSuccess) e = cudaFuncSetAttribute(epCombineRankReduceRecv, cudaFuncAttributeMaxDynamicSharedMemorySize, kRrCtaBytes);
            if (e != cudaSuccess) return e;
            attr_done[dev] = true;
        }
        const int want = 2 * (p.grid > 0 ? p.grid : sms); // p.grid counts SMs
        if (p.phases & 1) { // cooperative: its CTAs meet at a grid barrier before the flags go out
            const int grid = coopGrid(reinterpret_cast<const void *>(epCombineRankReduceSend), want, kRrCtaBytes);
            const cudaError_t e = cudaLaunchCooperativeKernel(reinterpret_cast<const void *>(epCombineRankReduceSend), dim3(grid), dim3(kThreads), args,
                                                              kRrCtaBytes, static_cast<cudaStream_t>(stream));
            if (e != cudaSuccess) return e;
        }
        if (p.phases & 2) {
            epCombineRankReduceRecv<<<want, kThreads, kRrCtaBytes, static_cast<cudaStream_t>(stream)>>>(p);
            return cudaGetLastError();
        }
        return cudaSuccess;
    }
    const int grid = coopGrid(reinterpret_cast<const void *>(epCombineKernel), p.grid, 0);
    return cudaLaunchCooperativeKernel(reinterpret_cast<const void *>(epCombineKernel), dim3(grid), dim3(kThreads), args, 0,
                                       static_cast<cudaStream_t>(stream));
}

extern "C" int nixl_ep_barrier_launch(const void *peers, int64_t off_flags, int32_t R, int32_t rank, uint64_t epoch, uint64_t timeout_ns,
                                      int32_t *status, int32_t *mask, void *stream) {
    if (!peers || R <= 0 || R > kMaxRanks || !status || !mask) return cudaErrorInvalidValue;
    epBarrierKernel<<<1, kMaxRanks, 0, static_cast<cudaStream_t>(stream)>>>(peers, off_flags, R, rank, epoch, timeout_ns, status, mask);
    return cudaGetLastError();
}

extern "C" int nixl_ep_layout_launch(const int64_t *topk_idx, int32_t T, int32_t K, int32_t E, int32_t R, int32_t *per_rank, int32_t *per_expert,
                                     uint8_t *in_rank, void *stream) {
    if (!topk_idx || !per_rank || !per_expert || !in_rank || T < 0 || K <= 0 || E <= 0 || R <= 0 || R > kMaxRanks || E % R) return cudaErrorInvalidValue;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    cudaError_t e = cudaMemsetAsync(per_rank, 0, sizeof(int32_t) * R, st);
    if (e == cudaSuccess) e = cudaMemsetAsync(per_expert, 0, sizeof(int32_t) * E, st);
    if (e != cudaSuccess) return e;
    if (T == 0) return cudaSuccess;
    const int blocks = (T + 255) / 256 < 148 ? (T + 255) / 256 : 148;
    epLayoutKernel<<<blocks, 256, sizeof(int) * (E + R), st>>>(topk_idx, T, K, E, R, per_rank, per_expert, in_rank);
    return cudaGetLastError();
}
