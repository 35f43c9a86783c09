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
// An entry >= n is skipped (its slot keeps its own item) and sets ST_RANGE.
#include <algorithm>

#include "rz_common.cuh"
#include "rz_internal.h"

namespace rz {

constexpr int kKeepIpt = 4;  // items per thread, all loads issued before any store

// One kept item. A load that misses L2 fetches its whole 128-byte line from DRAM unless it says
// otherwise; the kept items are far apart, so these ask for 64 bytes (4 sorted bytes out of every
// 256, 1 GiB: 442 -> 256 MB of DRAM reads, 68 -> 48 us) and do not stay in L1.
__device__ __forceinline__ uint32_t ld_sparse(const uint32_t* a) {
    uint32_t v;
    asm volatile("ld.global.L1::no_allocate.L2::64B.b32 %0, [%1];" : "=r"(v) : "l"(a) : "memory");
    return v;
}
__device__ __forceinline__ uint2 ld_sparse(const uint2* a) {
    uint2 v;
    asm volatile("ld.global.L1::no_allocate.L2::64B.v2.b32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "l"(a) : "memory");
    return v;
}
__device__ __forceinline__ uint4 ld_sparse(const uint4* a) {
    uint4 v;
    asm volatile("ld.global.L1::no_allocate.L2::64B.v4.b32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(a) : "memory");
    return v;
}
__device__ __forceinline__ u32x8 ld_sparse(const u32x8* a) {
    u32x8 v;
    v.a = ld_sparse(&a->a);
    v.b = ld_sparse(&a->b);
    return v;
}

template <int W>
__global__ void __launch_bounds__(256) keep_stage_kernel(const uint8_t* __restrict__ data, uint32_t n,
                                                         const uint32_t* __restrict__ keep, uint32_t m,
                                                         uint8_t* __restrict__ stage, uint32_t* status) {
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
        oor |= j < m && r[q] >= n;
    }
#pragma unroll
    for (int q = 0; q < kKeepIpt; ++q)
        if (r[q] < m) v[q] = ld_sparse(A + r[q]);
#pragma unroll
    for (int q = 0; q < kKeepIpt; ++q)
        if (r[q] < m) S[base + uint64_t(q) * 256] = v[q];
    if (oor) atomicOr(status, ST_RANGE);
}

// Bound by the random reads. n = 33.5M items of 16 bytes, m = 2.1M in order: a call takes 38.6 us;
// gathering all m items into the scratch with plain loads and copying it back took 59.2 us.
template <int W>
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
        if (r[q] < n) v[q] = ld_sparse(r[q] < m ? S + base + uint64_t(q) * 256 : A + r[q]);
#pragma unroll
    for (int q = 0; q < kKeepIpt; ++q)
        if (r[q] < n) st_item(A + base + uint64_t(q) * 256, v[q]);
}

template <int W>
static cudaError_t keep_launch(void* data, uint32_t n, const uint32_t* keep, uint32_t m, void* stage, uint32_t* status,
                        cudaStream_t s) {
    const uint32_t grid = uint32_t((uint64_t(m) + 256 * kKeepIpt - 1) / (256 * kKeepIpt));
    uint8_t* d = static_cast<uint8_t*>(data);
    uint8_t* st = static_cast<uint8_t*>(stage);
    const cudaError_t e = launch_pdl(keep_stage_kernel<W>, grid, 256, 0, s, d, n, keep, m, st, status);
    return e != cudaSuccess ? e : launch_pdl(keep_place_kernel<W>, grid, 256, 0, s, d, n, keep, m, st);
}

int launch_keep(rz_ctx* ctx, void* data, uint32_t n, uint32_t w, const uint32_t* keep, uint32_t m, void* stage,
                cudaStream_t s) {
    if (m == 0) return RZ_OK;
    switch (w) {
        case 4: RZ_CUDA_TRY(ctx, keep_launch<4>(data, n, keep, m, stage, ctx->ws.status, s)); break;
        case 8: RZ_CUDA_TRY(ctx, keep_launch<8>(data, n, keep, m, stage, ctx->ws.status, s)); break;
        case 16: RZ_CUDA_TRY(ctx, keep_launch<16>(data, n, keep, m, stage, ctx->ws.status, s)); break;
        default: RZ_CUDA_TRY(ctx, keep_launch<32>(data, n, keep, m, stage, ctx->ws.status, s)); break;
    }
    return RZ_OK;
}

}  // namespace rz
