// rz_keep.cu -- preserve-list compaction: data[0..m) = (old) data[keep[0..m)], O(m) work.
//
// The inverse form of removal that the paper names as future work: when the kept items are fewer
// than the removed ones, gathering them costs m random reads instead of the n - m moves a removal
// would make. In place in two kernels on the caller's stream. A write goes to [0, m) only, so an
// item kept from [m, n) can be read at any time; one kept from [0, m) may be overwritten by another
// slot and is copied to context scratch first:
//   stage:  stage[j] = data[keep[j]] for the entries with keep[j] < m (a share m / n of a list
//           without order or of a sorted one);
//   place:  data[j] = stage[j] for those, data[keep[j]] for all others.
// With more than seven eighths of the items kept, all of them are staged and copied back.
// An entry >= n is skipped (its slot keeps its own item) and sets ST_RANGE.
#include <algorithm>

#include "rz_common.cuh"
#include "rz_internal.h"

namespace rz {

constexpr int kKeepIpt = 4;  // items per thread, all loads issued before any store

// Which loads: plain ones through L2 (kNear), ones that ask for 64 bytes of a line that misses L2 instead of all of
// it (kFar), or those leaving nothing in L1 besides (kSparse). us a call, near / far / sparse, list in L2 as far as
// it fits. Far: in lists that are well past L2, kept items of 64 bytes and more apart (2^27 of 16 bytes, every 8th
// sorted 292 / 221 / 233, in random order 467 / 446 / 469); closer together or in shorter lists the rest of the line
// is wanted too (2^24 of 4 bytes, all in random order 114 / 120 / 188, a quarter of 50M 166 / 183 / 219). Sparse:
// among those, where the lines of the kept items are more than L2 holds and hardly any is used twice (2^27 of 4
// bytes, every 16th sorted 87 / 70 / 62, random 179 / 180 / 177; every 64th of 16 bytes sorted 54 / 48 / 42); such
// lines leave L2 early where they could stay (786k of 50M 11 / 11 / 18). With three lists in turn, so that L2 holds
// none, the gain is less and gone at every 16th of 16 bytes (2^25, sorted 33 / 35; one list 33 / 27).
enum KeepLoads { kNear, kFar, kSparse };
static KeepLoads keep_loads(uint32_t n, uint32_t m, uint32_t w) {
    const uint64_t bytes = uint64_t(n) * w;
    if (bytes < (192u << 20) || bytes < uint64_t(m) * 64) return kNear;
    return m >= (1u << 20) && n / (w < 16 ? 16 : 32) >= m && w < 32 ? kSparse : kFar;
}
// Nearly all items kept: they are all staged and copied back, which reads the list of entries once less (2^24 of 4
// bytes, all in random order: 103 us, 114 in two kernels; of 50M 752 / 783, three quarters of them 566 / 465).
static bool keep_all(uint32_t n, uint32_t m) { return m > n - n / 8; }

// One kept item. (4 sorted bytes out of every 256, 1 GiB, 128 / 64 bytes a miss: 442 / 256 MB of DRAM reads, 68 / 48
// us.)
template <KeepLoads L>
__device__ __forceinline__ uint32_t ld_kept(const uint32_t* a) {
    uint32_t v;
    if constexpr (L == kNear) v = ld_l2(a);
    else if constexpr (L == kFar) asm volatile("ld.global.cg.L2::64B.b32 %0, [%1];" : "=r"(v) : "l"(a) : "memory");
    else asm volatile("ld.global.L1::no_allocate.L2::64B.b32 %0, [%1];" : "=r"(v) : "l"(a) : "memory");
    return v;
}
template <KeepLoads L>
__device__ __forceinline__ uint2 ld_kept(const uint2* a) {
    uint2 v;
    if constexpr (L == kNear) v = ld_l2(a);
    else if constexpr (L == kFar)
        asm volatile("ld.global.cg.L2::64B.v2.b32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "l"(a) : "memory");
    else
        asm volatile("ld.global.L1::no_allocate.L2::64B.v2.b32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "l"(a) : "memory");
    return v;
}
template <KeepLoads L>
__device__ __forceinline__ uint4 ld_kept(const uint4* a) {
    uint4 v;
    if constexpr (L == kNear) v = ld_l2(a);
    else if constexpr (L == kFar)
        asm volatile("ld.global.cg.L2::64B.v4.b32 {%0, %1, %2, %3}, [%4];"
                     : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(a) : "memory");
    else
        asm volatile("ld.global.L1::no_allocate.L2::64B.v4.b32 {%0, %1, %2, %3}, [%4];"
                     : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(a) : "memory");
    return v;
}
// 32-byte items: one load of the whole sector where the list lies on 32 bytes. Elsewhere two that may meet
// in L1: past it they are two requests to L2 (2^23 of 2^27 in random order: 381 us, 262 with one).
template <KeepLoads L>
__device__ __forceinline__ u32x8 ld_kept(const u32x8* a) {
    if (!whole_sector(a)) return *a;
    u32x8 v;
    if constexpr (L != kNear)
        asm volatile("ld.global.L1::no_allocate.L2::64B.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                     : "=r"(v.a.x), "=r"(v.a.y), "=r"(v.a.z), "=r"(v.a.w), "=r"(v.b.x), "=r"(v.b.y), "=r"(v.b.z), "=r"(v.b.w)
                     : "l"(a) : "memory");
    else
        asm volatile("ld.global.L1::no_allocate.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                     : "=r"(v.a.x), "=r"(v.a.y), "=r"(v.a.z), "=r"(v.a.w), "=r"(v.b.x), "=r"(v.b.y), "=r"(v.b.z), "=r"(v.b.w)
                     : "l"(a) : "memory");
    return v;
}

// `cap`: n, and every item is staged, or m, and those kept from [0, m) are.
template <int W, KeepLoads L>
__global__ void __launch_bounds__(256) keep_stage_kernel(const uint8_t* data, uint32_t n, uint32_t cap,
                                                         const uint32_t* __restrict__ keep, uint32_t m,
                                                         uint8_t* stage, uint32_t* status) {
    using T = typename Payload<W>::T;
    pdl_begin();
    const T* A = reinterpret_cast<const T*>(data);
    T* S = reinterpret_cast<T*>(stage);
    bool oor = false;
    const uint64_t base = uint64_t(blockIdx.x) * (256 * kKeepIpt) + threadIdx.x;
    uint32_t r[kKeepIpt];
    T v[kKeepIpt];
#pragma unroll
    for (int q = 0; q < kKeepIpt; ++q) {
        const uint64_t j = base + uint64_t(q) * 256;
        r[q] = j < m ? ld_l2(&keep[j]) : 0xffffffffu;
    }
#pragma unroll
    for (int q = 0; q < kKeepIpt; ++q) {
        const uint64_t j = base + uint64_t(q) * 256;
        const bool past = j < m && r[q] >= n;
        oor |= past;
        r[q] = past && cap == n ? uint32_t(j) : r[q];  // all staged: the slot keeps its own item
    }
#pragma unroll
    for (int q = 0; q < kKeepIpt; ++q)
        if (r[q] < cap) v[q] = ld_kept<L>(A + r[q]);
#pragma unroll
    for (int q = 0; q < kKeepIpt; ++q)
        if (r[q] < cap) S[base + uint64_t(q) * 256] = v[q];
    if (oor) atomicOr(status, ST_RANGE);
}

// Bound by the random reads. n = 33.5M items of 16 bytes, m = 2.1M in order: a call takes 33 us;
// gathering all m items into the scratch with plain loads and copying it back took 59.
template <int W, KeepLoads L>
__global__ void __launch_bounds__(256) keep_place_kernel(uint8_t* data, uint32_t n, const uint32_t* __restrict__ keep,
                                                         uint32_t m, const uint8_t* __restrict__ stage) {
    using T = typename Payload<W>::T;
    pdl_begin();
    T* A = reinterpret_cast<T*>(data);
    const T* S = reinterpret_cast<const T*>(stage);
    const uint64_t base = uint64_t(blockIdx.x) * (256 * kKeepIpt) + threadIdx.x;
    uint32_t r[kKeepIpt];
    T v[kKeepIpt];
#pragma unroll
    for (int q = 0; q < kKeepIpt; ++q) {
        const uint64_t j = base + uint64_t(q) * 256;
        r[q] = j < m ? ld_l2(&keep[j]) : 0xffffffffu;
    }
#pragma unroll
    for (int q = 0; q < kKeepIpt; ++q)
        if (r[q] < n) v[q] = ld_kept<L>(r[q] < m ? S + base + uint64_t(q) * 256 : A + r[q]);
#pragma unroll
    for (int q = 0; q < kKeepIpt; ++q)
        if (r[q] < n) st_item(A + base + uint64_t(q) * 256, v[q]);
}

template <int W, KeepLoads L>
static cudaError_t keep_launch(void* data, uint32_t n, const uint32_t* keep, uint32_t m, void* stage, uint32_t* status,
                        cudaStream_t s) {
    const uint32_t grid = uint32_t((uint64_t(m) + 256 * kKeepIpt - 1) / (256 * kKeepIpt));
    uint8_t* d = static_cast<uint8_t*>(data);
    uint8_t* st = static_cast<uint8_t*>(stage);
    const bool all = keep_all(n, m);
    const cudaError_t e = launch_pdl(keep_stage_kernel<W, L>, grid, 256, 0, s, d, n, all ? n : m, keep, m, st, status);
    if (e != cudaSuccess) return e;
    if (all) return cudaMemcpyAsync(data, stage, size_t(m) * W, cudaMemcpyDeviceToDevice, s);
    return launch_pdl(keep_place_kernel<W, L>, grid, 256, 0, s, d, n, keep, m, st);
}

using KeepFn = cudaError_t (*)(void*, uint32_t, const uint32_t*, uint32_t, void*, uint32_t*, cudaStream_t);
template <int W>
static KeepFn keep_launch(KeepLoads l) {
    if constexpr (W == 32) return l == kNear ? keep_launch<W, kNear> : keep_launch<W, kFar>;
    else return l == kNear ? keep_launch<W, kNear> : l == kFar ? keep_launch<W, kFar> : keep_launch<W, kSparse>;
}

int launch_keep(rz_ctx* ctx, void* data, uint32_t n, uint32_t w, const uint32_t* keep, uint32_t m, void* stage,
                cudaStream_t s) {
    if (m == 0) return RZ_OK;
    const KeepLoads l = keep_loads(n, m, w);
    const auto f = w == 4    ? keep_launch<4>(l)
                   : w == 8  ? keep_launch<8>(l)
                   : w == 16 ? keep_launch<16>(l)
                             : keep_launch<32>(l);
    RZ_CUDA_TRY(ctx, f(data, n, keep, m, stage, ctx->ws.status, s));
    ctx->last_kernels = keep_all(n, m) ? 1 : 2;
    return RZ_OK;
}

}  // namespace rz
