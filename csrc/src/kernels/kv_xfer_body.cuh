// Device-side body of the paged KV-cache transfer, shared by the regular entry point
// (kv_xfer.cu: block tables and completion counter in caller-provided device memory) and the
// allocation-free one (kv_xfer_static.cu: both inside the library's own scratch area).
//
// Work unit: a warp's step of kSlots slots, a slot being 32 consecutive vectors (one per lane, 32 source bytes where rows,
// strides and addresses allow, else 16) of one (cache tensor, block pair).  The kernel is bound by memory: what it needs is
// bytes in flight all the time and an even split.
//   - 32 resident warps per SM with 2 x 1 KiB each keep 64 KiB per SM in flight; all CTAs together walk one window of
//     consecutive blocks.  More in flight is slower, not faster (the first shape below: 50.8 - 51.6 us with 32 to 64 KiB per
//     SM, 53.2 with 128, 60.7 with 96 in 48 warps), and so are CTAs that each walk a range of their own (55 - 58 us).
//   - A request is split in steps of 2 KiB, so that the last round of a short one is nearly as full as the others (the
//     second shape made 732 groups for 592 CTAs when a CTA took four whole blocks: two rounds for 1.24).
//   - Where a step's bytes lie takes a chain of loads (block table, view entry).  One lane per slot looks the next step's
//     slots up while the loads of this one are in flight.
//   - Rows that are contiguous on both sides are merged on the host, and indexes divide by multiplication.
// Measured on one B200 (bytes read + written, before / now): 64 tensors x 256 blocks of 8 KiB, bf16, 268 MB: 54.2 / 51.6 us
// (5.2 TB/s); 48 tensors x 61 blocks of 16 KiB, fp8 cast and token-major to head-major, 72 MB: 22.4 / 18.9 us (3.8 TB/s), with the one
// in front overlapped; each kilobyte read is then stored as eight pieces of 64 bytes, as blocks are walked in the source's order.
#ifndef NIXL_B200_KV_XFER_BODY_CUH
#define NIXL_B200_KV_XFER_BODY_CUH

#include <cuda_bf16.h>
#include <cuda_fp8.h>
#include <cuda_runtime.h>

#include "device/nixl_device_layout.h"
#include "kernels/nixl_kernels.h"

namespace nixl_kv {

constexpr int kKvThreads = 256;
constexpr int kSlots = 2; // slots in flight per warp

// n / d for n < 2^31 by a multiplication.
struct FastDiv {
    uint32_t d, m, s;
    __device__ __forceinline__ uint32_t quot(uint32_t n) const { return (__umulhi(n, m) + n) >> s; }
};
inline FastDiv fastDiv(uint32_t d) {
    const uint32_t s = d > 1 ? 32 - __builtin_clz(d - 1) : 0; // ceil(log2 d)
    return {d, static_cast<uint32_t>((((uint64_t(1) << s) - d) << 32) / d + 1), s};
}

// What the kernels work from: the request with its contiguous rows merged and its divisors prepared.
struct KvPlan {
    NixlKvXferParams p;
    int64_t src_token_stride, src_head_stride, dst_token_stride, dst_head_stride; // of the merged rows
    FastDiv vec_per_row, heads;  // vectors per merged row, merged rows per token
    uint32_t vec_per_unit;
    uint32_t parts;              // slots per (tensor, block pair)
    FastDiv parts_div, pairs_div;
    long long slots;             // of the whole request
    int vec_bytes;               // 32 or 16 source bytes per vector
};

inline KvPlan planFor(const NixlKvXferParams &p) {
    KvPlan k{};
    k.p = p;
    const int shrink = p.cast_fp8 ? 2 : 1;
    int64_t row = p.head_bytes, tokens = p.tokens, heads = p.heads;
    for (int pass = 0; pass < 2; ++pass) { // heads into the row, tokens into the row, in whichever order they are contiguous
        if (heads > 1 && p.src_head_stride == row && p.dst_head_stride * shrink == row) {
            row *= heads;
            heads = 1;
        }
        if (tokens > 1 && p.src_token_stride == row && p.dst_token_stride * shrink == row) {
            row *= tokens;
            tokens = 1;
        }
    }
    const int64_t sa = p.src_block_stride | (tokens > 1 ? p.src_token_stride : 0) | (heads > 1 ? p.src_head_stride : 0);
    const int64_t da = p.dst_block_stride | (tokens > 1 ? p.dst_token_stride : 0) | (heads > 1 || p.dst_head_offset ? p.dst_head_stride : 0);
    k.vec_bytes = (row % 32 == 0 && sa % 32 == 0 && da % (32 / shrink) == 0) ? 32 : 16;
    k.src_token_stride = p.src_token_stride;
    k.src_head_stride = p.src_head_stride;
    k.dst_token_stride = p.dst_token_stride;
    k.dst_head_stride = p.dst_head_stride;
    k.vec_per_row = fastDiv(static_cast<uint32_t>(row / k.vec_bytes));
    k.heads = fastDiv(static_cast<uint32_t>(heads));
    k.vec_per_unit = static_cast<uint32_t>(tokens * heads * (row / k.vec_bytes));
    k.parts = (k.vec_per_unit + 31) / 32;
    k.parts_div = fastDiv(k.parts);
    k.pairs_div = fastDiv(static_cast<uint32_t>(p.n_pairs));
    k.slots = static_cast<long long>(p.n_tensors) * p.n_pairs * k.parts;
    return k;
}

// A block id.  Volatile, and not through the read-only path: the kernel in front may write the tables while this one's CTAs wait
// for it, and nothing else keeps the load behind that wait.
__device__ __forceinline__ int32_t ldBlock(const int32_t *p) {
    int32_t b;
    asm volatile("ld.global.s32 %0, [%1];" : "=r"(b) : "l"(p));
    return b;
}
__device__ __forceinline__ uint4 ldStream(const void *p) {
    uint4 v;
    asm volatile("ld.global.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
    return v;
}
__device__ __forceinline__ void ldStream32(const void *p, uint4 &lo, uint4 &hi) {
    asm volatile("ld.global.L1::no_allocate.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(lo.x), "=r"(lo.y), "=r"(lo.z), "=r"(lo.w), "=r"(hi.x), "=r"(hi.y), "=r"(hi.z), "=r"(hi.w)
                 : "l"(p));
}
__device__ __forceinline__ void stStream16(void *p, const uint4 &v) {
    asm volatile("st.global.L1::no_allocate.v4.u32 [%0], {%1,%2,%3,%4};" ::"l"(p), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}
__device__ __forceinline__ void stStream32(void *p, const uint4 &lo, const uint4 &hi) {
    asm volatile("st.global.L1::no_allocate.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(p), "r"(lo.x), "r"(lo.y), "r"(lo.z), "r"(lo.w), "r"(hi.x),
                 "r"(hi.y), "r"(hi.z), "r"(hi.w)
                 : "memory");
}
__device__ __forceinline__ void stStream8(void *p, const uint2 &v) {
    asm volatile("st.global.L1::no_allocate.v2.u32 [%0], {%1,%2};" ::"l"(p), "r"(v.x), "r"(v.y) : "memory");
}

// Two bf16 (packed in a u32) -> two e4m3 (packed in the low 16 bits), after scaling.
__device__ __forceinline__ uint32_t castPair(uint32_t packed, float scale) {
    const __nv_bfloat162 b = *reinterpret_cast<const __nv_bfloat162 *>(&packed);
    float2 f = __bfloat1622float2(b);
    f.x *= scale;
    f.y *= scale;
    return static_cast<uint32_t>(__nv_cvt_float2_to_fp8x2(f, __NV_SATFINITE, __NV_E4M3));
}

__device__ __forceinline__ uint2 castVec(const uint4 &v, float scale) {
    uint2 o;
    o.x = castPair(v.x, scale) | (castPair(v.y, scale) << 16);
    o.y = castPair(v.z, scale) | (castPair(v.w, scale) << 16);
    return o;
}

// Where one slot's block starts on both sides (null: nothing to move) and its first vector.
struct SlotRef {
    const char *src;
    char *dst;
    uint32_t vec0;
};

__device__ __forceinline__ SlotRef lookUp(const KvPlan &k, const int32_t *src_blocks, const int32_t *dst_blocks, long long slot) {
    SlotRef r{nullptr, nullptr, 0};
    if (slot >= k.slots) return r;
    const NixlKvXferParams &p = k.p;
    const nixlMemViewEntry *src_ent = reinterpret_cast<const nixlMemViewEntry *>(static_cast<const char *>(p.src_view) + sizeof(nixlMemViewHeader));
    const nixlMemViewEntry *dst_ent = reinterpret_cast<const nixlMemViewEntry *>(static_cast<const char *>(p.dst_view) + sizeof(nixlMemViewHeader));
    // Pairs vary fastest so that consecutive units read one tensor's blocks.
    uint32_t part, t, i;
    if (k.slots <= 0x7fffffffll) {
        const uint32_t u = k.parts_div.quot(static_cast<uint32_t>(slot));
        part = static_cast<uint32_t>(slot) - u * k.parts;
        t = k.pairs_div.quot(u);
        i = u - t * static_cast<uint32_t>(p.n_pairs);
    } else {
        const long long u = slot / k.parts;
        part = static_cast<uint32_t>(slot - u * k.parts);
        t = static_cast<uint32_t>(u / p.n_pairs);
        i = static_cast<uint32_t>(u - static_cast<long long>(t) * p.n_pairs);
    }
    // Bytes a block spans from its base on either side (strides are non-negative), for the bounds check.
    const long long src_extent = (p.tokens - 1LL) * p.src_token_stride + (p.heads - 1LL) * p.src_head_stride + p.head_bytes;
    const long long dst_extent = (p.tokens - 1LL) * p.dst_token_stride + (p.dst_head_offset + p.heads - 1LL) * p.dst_head_stride +
        (p.cast_fp8 ? p.head_bytes / 2 : p.head_bytes);
    const long long sb = ldBlock(src_blocks + i), db = ldBlock(dst_blocks + i);
    const long long soff = sb * p.src_block_stride, doff = db * p.dst_block_stride;
    // The block tables come from device memory that nobody validated: a block must lie inside its tensor's
    // registered range on both sides, or it is skipped and reported.
    const bool inside = sb >= 0 && db >= 0 && src_ent[t].ptr != 0 && dst_ent[t].ptr != 0 &&
        static_cast<unsigned long long>(soff + src_extent) <= src_ent[t].len && static_cast<unsigned long long>(doff + dst_extent) <= dst_ent[t].len;
    if (inside) {
        r.src = reinterpret_cast<const char *>(src_ent[t].ptr) + soff;
        r.dst = reinterpret_cast<char *>(dst_ent[t].ptr) + doff + static_cast<long long>(p.dst_head_offset) * p.dst_head_stride;
        r.vec0 = part * 32;
    } else if (p.status != nullptr) {
        *reinterpret_cast<volatile int32_t *>(p.status) = 1;
    }
    return r;
}

// Moves every (tensor, block pair) unit of the request.  src_blocks / dst_blocks are the block
// tables in device memory (wherever the entry point keeps them).
template<bool kCast, int kVec>
__device__ __forceinline__ void moveBlocks(const KvPlan &k, const int32_t *src_blocks, const int32_t *dst_blocks) {
    constexpr int kDstVec = kCast ? kVec / 2 : kVec;
    const unsigned lane = threadIdx.x & 31u;
    const long long warps = static_cast<long long>(gridDim.x) * (kKvThreads / 32);
    long long first = (static_cast<long long>(blockIdx.x) * (kKvThreads / 32) + (threadIdx.x >> 5)) * kSlots;
    SlotRef cur{nullptr, nullptr, 0};
    if (lane < kSlots) cur = lookUp(k, src_blocks, dst_blocks, first + lane);
    for (; first < k.slots; first += warps * kSlots) { // uniform over the warp
        uint4 lo[kSlots], hi[kSlots];
        char *to[kSlots];
        bool wide[kSlots];
#pragma unroll
        for (int j = 0; j < kSlots; ++j) {
            const char *sbase = reinterpret_cast<const char *>(__shfl_sync(0xffffffffu, reinterpret_cast<unsigned long long>(cur.src), j));
            char *dbase = reinterpret_cast<char *>(__shfl_sync(0xffffffffu, reinterpret_cast<unsigned long long>(cur.dst), j));
            const uint32_t vec = __shfl_sync(0xffffffffu, cur.vec0, j) + lane;
            const bool here = sbase != nullptr && vec < k.vec_per_unit;
            const uint32_t at = here ? vec : 0;
            const uint32_t row = k.vec_per_row.quot(at), v = at - row * k.vec_per_row.d;
            const uint32_t token = k.heads.quot(row), head = row - token * k.heads.d;
            const char *from = sbase + token * k.src_token_stride + head * k.src_head_stride + static_cast<size_t>(v) * kVec;
            to[j] = here ? dbase + token * k.dst_token_stride + head * k.dst_head_stride + static_cast<size_t>(v) * kDstVec : nullptr;
            // a cache tensor may start at any multiple of 16 bytes (8 for the cast's destination)
            wide[j] = kVec == 32 && ((reinterpret_cast<uintptr_t>(sbase) & 31) | (reinterpret_cast<uintptr_t>(dbase) & (kDstVec - 1))) == 0;
            lo[j] = hi[j] = make_uint4(0, 0, 0, 0);
            if (here) {
                if (kVec == 32 && wide[j]) {
                    ldStream32(from, lo[j], hi[j]);
                } else {
                    lo[j] = ldStream(from);
                    if constexpr (kVec == 32) hi[j] = ldStream(from + 16);
                }
            }
        }
        if (lane < kSlots) cur = lookUp(k, src_blocks, dst_blocks, first + warps * kSlots + lane); // behind the loads in flight
#pragma unroll
        for (int j = 0; j < kSlots; ++j) {
            if (to[j] == nullptr) continue;
            if constexpr (kCast) {
                const uint2 a = castVec(lo[j], k.p.scale);
                if constexpr (kVec == 32) {
                    const uint2 b = castVec(hi[j], k.p.scale);
                    if (wide[j]) {
                        stStream16(to[j], make_uint4(a.x, a.y, b.x, b.y));
                    } else {
                        stStream8(to[j], a);
                        stStream8(to[j] + 8, b);
                    }
                } else {
                    stStream8(to[j], a);
                }
            } else if (kVec == 32 && wide[j]) {
                stStream32(to[j], lo[j], hi[j]);
            } else {
                stStream16(to[j], lo[j]);
                if constexpr (kVec == 32) stStream16(to[j] + 16, hi[j]);
            }
        }
    }
}

// Completion: the last CTA to finish signals the receiver (and the host, if asked).  One
// acquire-release add at GPU scope chains the CTAs; the release operations at system scope
// that follow publish every CTA's stores before the signal becomes visible.  `counter` is zero
// before the launch and is left at zero.
__device__ __forceinline__ void signalWhenAllDone(const NixlKvXferParams &p, unsigned int *counter) {
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned prev;
        asm volatile("atom.add.acq_rel.gpu.global.u32 %0, [%1], 1;" : "=r"(prev) : "l"(counter) : "memory");
        if (prev == gridDim.x - 1) {
            *counter = 0;
            if (p.done_signal) asm volatile("red.release.sys.global.add.u64 [%0], %1;" ::"l"(p.done_signal), "l"(p.done_value) : "memory");
            if (p.host_flag) asm volatile("st.release.sys.global.u64 [%0], %1;" ::"l"(p.host_flag), "l"(p.host_seq) : "memory");
        }
    }
}

// Grid for a request: `wanted`, or by default four CTAs per SM of the current device, what is resident at once, and twice as
// many when every warp has sixteen steps or more (the second half then starts staggered: 72 tensors x 195 blocks of 16 KiB
// 78.9 us against 83.6, 72 x 164 of 24 KiB 100 against 107; 48 x 61 of 16 KiB, five steps per warp, 20.6 against 18.7).
// Never more than there are steps for: CTAs without any would only lengthen the completion count.
inline int gridFor(const KvPlan &k, int device) {
    static int sm_count[64] = {}; // per device, looked up once (this is the post path)
    int grid = k.p.grid;
    const long long want = (k.slots + kSlots - 1) / kSlots;
    if (grid <= 0) {
        int sms = device >= 0 && device < 64 ? sm_count[device] : 0;
        if (sms <= 0) {
            if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess || sms <= 0) sms = 148;
            if (device >= 0 && device < 64) sm_count[device] = sms;
        }
        grid = sms * 4;
        if (want >= 16LL * grid * (kKvThreads / 32)) grid *= 2;
    }
    const long long most = (want + kKvThreads / 32 - 1) / (kKvThreads / 32);
    return grid > most ? static_cast<int>(most) : grid;
}

// Shape and alignment checks common to both entry points; cudaSuccess when the request is well formed.
inline cudaError_t checkShape(const NixlKvXferParams &p) {
    if (p.n_pairs <= 0 || p.n_tensors <= 0 || p.tokens <= 0 || p.heads <= 0 || p.head_bytes <= 0 || (p.head_bytes & 15))
        return cudaErrorInvalidValue;
    // Vector accesses need 16-byte (8-byte when casting) aligned strides.
    const int64_t sa = p.src_block_stride | p.src_token_stride | p.src_head_stride;
    const int64_t da = p.dst_block_stride | p.dst_token_stride | p.dst_head_stride;
    if ((sa & 15) || (da & (p.cast_fp8 ? 7 : 15))) return cudaErrorInvalidValue;
    return cudaSuccess;
}

} // namespace nixl_kv

#endif
