// rz_keyidx.cu -- a key -> row index kept current under Redzone moves, for delete-by-key.
//
// Records are 8, 16 or 32 bytes and start with a uint64 key (two reserved values: all ones marks
// an empty slot, all ones minus one an erased one). The index is an open-addressing hash table on
// the device: capacity a power of two, linear probing from the SplitMix64 finaliser of the key
// (Steele, Lea and Flood, "Fast splittable pseudorandom number generators", 2014).
//
// Removal by key keeps the index exact in O(k): the canonical rule moves an item only into a hole
// below the cut (every other surviving item keeps its row), so after the removal each hole's new
// occupant is re-pointed at the hole, and the deleted keys are erased. Nothing is rescanned.
// The lookup also claims the row of each key (one bit of the map that RZ_VALIDATE uses), which catches a key
// given twice and two keys of one row; it takes the place of RZ_VALIDATE's passes. What it finds wrong
// goes into the context's status word, which the removal (as after those passes) and the index
// update look at before they change anything. So the whole call is queued at once and the host
// waits for it once. Bound by the random accesses of the probes and by that wait: deleting 65521 of
// 4.2M 32-byte records by key, inserting as many and looking as many up takes 67 us, and took 155 us
// with a wait after the lookup, validation passes over the rows, and 64-bit rows made from 32-bit ones
// by the caller. (Keys and rows in one 16-byte slot made the calls 7 % faster but the build slower by
// half: 134 MB of slots do not stay in L2.)
#include <algorithm>
#include <new>

#include "rz_common.cuh"
#include "rz_internal.h"

namespace rz {

constexpr unsigned long long kEmptyKey = ~0ull;
constexpr unsigned long long kErasedKey = ~0ull - 1ull;
constexpr uint32_t kNoRow = 0xffffffffu;
enum : uint32_t { IX_DUPLICATE = 1u, IX_FULL = 4u, IX_RESERVED = 8u };  // status bits of an insert

__device__ __forceinline__ unsigned long long mix64(unsigned long long z) {
    z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
    z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
    return z ^ (z >> 31);
}

__device__ __forceinline__ unsigned long long record_key(const uint8_t* data, uint32_t w, uint32_t row) {
    return *reinterpret_cast<const unsigned long long*>(data + size_t(row) * w);
}

// Slot holding `key`, or kNoRow (stops at the first empty slot; erased slots are passed over).
__device__ __forceinline__ uint32_t find_slot(const unsigned long long* keys, uint32_t mask, unsigned long long key) {
    uint32_t s = uint32_t(mix64(key)) & mask;
    for (uint32_t probe = 0; probe <= mask; ++probe, s = (s + 1u) & mask) {
        const unsigned long long k0 = keys[s];
        if (k0 == key) return s;
        if (k0 == kEmptyKey) return kNoRow;
    }
    return kNoRow;
}

__global__ void ix_insert_kernel(unsigned long long* keys, uint32_t* rows, uint32_t mask, const uint8_t* data,
                                 uint32_t w, uint32_t first, uint32_t count, uint32_t* status) {
    pdl_begin();
    for (uint32_t q = blockIdx.x * blockDim.x + threadIdx.x; q < count; q += gridDim.x * blockDim.x) {
        const uint32_t row = first + q;
        const unsigned long long key = record_key(data, w, row);
        if (key >= kErasedKey) {
            atomicOr(status, IX_RESERVED);
            continue;
        }
        uint32_t s = uint32_t(mix64(key)) & mask;
        bool done = false;
        for (uint32_t probe = 0; probe <= mask && !done; ++probe, s = (s + 1u) & mask) {
            unsigned long long k0 = keys[s];
            while (k0 == kEmptyKey || k0 == kErasedKey) {
                const unsigned long long prev = atomicCAS(&keys[s], k0, key);
                if (prev == k0) {
                    rows[s] = row;
                    done = true;
                    break;
                }
                k0 = prev;  // someone else took the slot: look at what they put there
            }
            if (!done && k0 == key) {
                atomicOr(status, IX_DUPLICATE);
                done = true;
            }
        }
        if (!done) atomicOr(status, IX_FULL);
    }
}

// Rows of the keys asked for; when absent kNoRow, or -1 in 64 bits.
template <typename Row>
__global__ void ix_find_kernel(const unsigned long long* keys, const uint32_t* rows, uint32_t mask,
                               const unsigned long long* q, uint32_t count, Row* out_rows) {
    pdl_begin();
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < count; i += gridDim.x * blockDim.x) {
        const unsigned long long key = q[i];
        const uint32_t s = key >= kErasedKey ? kNoRow : find_slot(keys, mask, key);
        out_rows[i] = s == kNoRow ? Row(-1) : Row(rows[s]);
    }
}

// Rows and slots of the keys to delete (kNoRow when absent); every row is claimed (seen: one bit per
// row of the list, zero before). A missing key, or one whose row is past the list, is an entry
// outside it (ST_RANGE); a key given twice, or two keys that lead to one row, a duplicate. An earlier
// call's error that is still in the status word refuses the call (ST_REFUSED): the index update goes by
// the whole word, so the removal must not go by a part of it.
__global__ void ix_claim_kernel(const unsigned long long* keys, const uint32_t* rows, uint32_t* seen, uint32_t mask,
                                const unsigned long long* q, uint32_t count, uint32_t n, uint32_t* out_rows,
                                uint32_t* out_slots, uint32_t* status) {
    pdl_begin();
    if (blockIdx.x == 0 && threadIdx.x == 0 && (__ldcg(status) & ~(ST_DUPLICATE | ST_RANGE)) != 0u)
        atomicOr(status, ST_REFUSED);
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < count; i += gridDim.x * blockDim.x) {
        const unsigned long long key = q[i];
        const uint32_t s = key >= kErasedKey ? kNoRow : find_slot(keys, mask, key);
        const uint32_t row = s == kNoRow ? kNoRow : rows[s];
        if (row >= n) {
            atomicOr(status, ST_RANGE);
        } else {
            const uint32_t bit = 1u << (row & 31u);
            if (atomicOr(&seen[row >> 5], bit) & bit) atomicOr(status, ST_DUPLICATE);
        }
        out_rows[i] = row;
        out_slots[i] = s;
    }
}

// After the removal, if it took place: erase the deleted keys, and point the key of the item that
// moved into each hole below the cut at the hole (a live key, so its probe never ends at a slot
// that is erased meanwhile).
__global__ void ix_update_kernel(unsigned long long* keys, uint32_t* rows, uint32_t* seen, uint32_t mask,
                                 const uint8_t* data, uint32_t w, const uint32_t* holes, const uint32_t* del_slots,
                                 uint32_t count, uint32_t cut, const uint32_t* status) {
    pdl_begin();
    if (__ldcg(status) != 0u) return;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < count; i += gridDim.x * blockDim.x) {
        const uint32_t h = holes[i], d = del_slots[i];
        keys[d] = kErasedKey;
        seen[h >> 5] = 0u;  // every claim in the word is this call's
        if (h >= cut) continue;
        const uint32_t s = find_slot(keys, mask, record_key(data, w, h));
        if (s != kNoRow) rows[s] = h;
    }
}

// A removal that did not take place lets go of its rows.
__global__ void ix_unclaim_kernel(uint32_t* seen, const uint32_t* del_rows, uint32_t count, uint32_t n) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < count; i += gridDim.x * blockDim.x)
        if (del_rows[i] < n) seen[del_rows[i] >> 5] = 0u;
}

static uint32_t grid_for(const rz_ctx* ctx, int64_t count) {
    return uint32_t(std::max<int64_t>(1, std::min<int64_t>(int64_t(ctx->sms) * 8, (count + 255) / 256)));
}

}  // namespace rz

struct rz_keyindex {
    rz_ctx* ctx = nullptr;
    unsigned long long* keys = nullptr;
    uint32_t* rows = nullptr;
    uint32_t mask = 0;
    uint32_t* status = nullptr;      // device
    uint32_t* del_rows = nullptr;    // removal list of the current call
    uint32_t* del_slots = nullptr;
    uint32_t* del_own = nullptr;     // their own allocation, once a removal outgrew the index's
    size_t del_cap = 0;
};

using namespace rz;

static int ix_status(rz_keyindex* ix, cudaStream_t s, uint32_t* bits) {
    int st = queue_status(ix->ctx, s, ix->status);
    if (st == RZ_OK) st = await_status(ix->ctx, s, bits);
    if (st != RZ_OK) return st;
    if (*bits) RZ_CUDA_TRY(ix->ctx, cudaMemsetAsync(ix->status, 0, 4, s));
    return RZ_OK;
}

static int ix_map(uint32_t bits) {
    if (bits & IX_RESERVED) return RZ_ERR_INVALID_ARG;
    if (bits & IX_FULL) return RZ_ERR_NO_MEMORY;
    if (bits & IX_DUPLICATE) return RZ_ERR_DUPLICATE;
    return RZ_OK;
}

template <typename Row>
static int ix_find(rz_keyindex* ix, const uint64_t* d_keys, int64_t count, Row* d_rows, rz_stream_t stream) {
    if (!ix || count < 0 || (count > 0 && (!d_keys || !d_rows)) || count > (int64_t(1) << 32) - 1)
        return RZ_ERR_INVALID_ARG;
    rz_ctx* ctx = ix->ctx;
    std::lock_guard<std::recursive_mutex> lock(ctx->mu);
    cudaSetDevice(ctx->device);
    if (count == 0) return RZ_OK;
    RZ_CUDA_TRY(ctx, launch_pdl(ix_find_kernel<Row>, grid_for(ctx, count), 256, 0, reinterpret_cast<cudaStream_t>(stream),
                                ix->keys, ix->rows, ix->mask, reinterpret_cast<const unsigned long long*>(d_keys),
                                uint32_t(count), d_rows));
    return RZ_OK;
}

static bool key_record(uint32_t w) { return w == 8 || w == 16 || w == 32; }

extern "C" {

int rz_keyindex_create(rz_ctx* ctx, int64_t capacity, rz_keyindex** out) {
    if (!ctx || !out || capacity < 1 || capacity > (int64_t(1) << 31)) return RZ_ERR_INVALID_ARG;
    std::lock_guard<std::recursive_mutex> lock(ctx->mu);
    cudaSetDevice(ctx->device);
    uint64_t cap = 2;
    while (cap < uint64_t(capacity)) cap <<= 1;
    rz_keyindex* ix = new (std::nothrow) rz_keyindex();
    if (!ix) return RZ_ERR_NO_MEMORY;
    ix->ctx = ctx;
    ix->mask = uint32_t(cap - 1);
    // Keys, and in a second allocation: rows | status | rows and slots of a removal of up to cap / 32
    // keys (a longer one gets arrays of its own; 2 % of the index). The removal list starts on 16
    // bytes, as the scanning schedules want it.
    const size_t row_words = size_t(cap + 3) & ~size_t(3);
    const size_t del = std::max<size_t>(size_t(cap / 32), 1024);
    cudaError_t e = cudaMalloc(&ix->keys, cap * 8);
    if (e == cudaSuccess) e = cudaMalloc(&ix->rows, (row_words + 4 + 2 * del) * 4);
    if (e == cudaSuccess) {
        ix->status = ix->rows + row_words;
        ix->del_rows = ix->status + 4;
        ix->del_slots = ix->del_rows + del;
        ix->del_cap = del;
        e = cudaMemset(ix->status, 0, 16);
    }
    if (e == cudaSuccess) e = cudaMemset(ix->keys, 0xff, cap * 8);
    if (e != cudaSuccess) {
        const int st = cuda_fail(ctx, e, "rz_keyindex_create");
        cudaFree(ix->keys);
        cudaFree(ix->rows);
        delete ix;
        return st;
    }
    *out = ix;
    return RZ_OK;
}

void rz_keyindex_destroy(rz_keyindex* ix) {
    if (!ix) return;
    cudaSetDevice(ix->ctx->device);
    cudaFree(ix->keys);
    cudaFree(ix->rows);
    cudaFree(ix->del_own);
    delete ix;
}

int rz_keyindex_insert(rz_keyindex* ix, const void* d_data, int64_t first, int64_t count, uint32_t record_bytes,
                       rz_stream_t stream) {
    if (!ix || !key_record(record_bytes) || first < 0 || count < 0 || first + count > (int64_t(1) << 32) - 1 ||
        (count > 0 && !d_data))
        return RZ_ERR_INVALID_ARG;
    rz_ctx* ctx = ix->ctx;
    std::lock_guard<std::recursive_mutex> lock(ctx->mu);
    cudaSetDevice(ctx->device);
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    if (count > 0) {
        RZ_CUDA_TRY(ctx, launch_pdl(ix_insert_kernel, grid_for(ctx, count), 256, 0, s, ix->keys, ix->rows, ix->mask,
                                    static_cast<const uint8_t*>(d_data), record_bytes, uint32_t(first), uint32_t(count),
                                    ix->status));
    }
    uint32_t bits = 0;
    const int st = ix_status(ix, s, &bits);
    return st != RZ_OK ? st : ix_map(bits);
}

int rz_keyindex_build(rz_keyindex* ix, const void* d_data, int64_t n, uint32_t record_bytes, rz_stream_t stream) {
    if (!ix) return RZ_ERR_INVALID_ARG;
    rz_ctx* ctx = ix->ctx;
    {
        std::lock_guard<std::recursive_mutex> lock(ctx->mu);
        cudaSetDevice(ctx->device);
        RZ_CUDA_TRY(ctx, cudaMemsetAsync(ix->keys, 0xff, (size_t(ix->mask) + 1) * 8,
                                         reinterpret_cast<cudaStream_t>(stream)));
    }
    return rz_keyindex_insert(ix, d_data, 0, n, record_bytes, stream);
}

int rz_keyindex_find(rz_keyindex* ix, const uint64_t* d_keys, int64_t count, uint32_t* d_rows, rz_stream_t stream) {
    return ix_find(ix, d_keys, count, d_rows, stream);
}

int rz_keyindex_find64(rz_keyindex* ix, const uint64_t* d_keys, int64_t count, int64_t* d_rows, rz_stream_t stream) {
    return ix_find(ix, d_keys, count, d_rows, stream);
}

int rz_remove_by_key(rz_ctx* ctx, rz_keyindex* ix, void* d_data, int64_t n, uint32_t record_bytes,
                     const uint64_t* d_keys, int64_t k, int64_t* new_len, uint32_t flags, rz_stream_t stream) {
    if (!ctx || !ix || ix->ctx != ctx || !key_record(record_bytes) || n < 0 || k < 0 || k > n ||
        n >= (int64_t(1) << 32) || (k > 0 && (!d_keys || !d_data)))
        return RZ_ERR_INVALID_ARG;
    std::lock_guard<std::recursive_mutex> lock(ctx->mu);
    cudaSetDevice(ctx->device);
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    if (new_len) *new_len = n - k;
    if (k == 0) return RZ_OK;
    // The index follows the Redzone rule only: the O(n) path would move rows that it does not look at.
    flags &= ~uint32_t(RZ_FORCE_PARTITION | RZ_ALLOW_STABLE);
    if (size_t(k) > ix->del_cap) {
        cudaFree(ix->del_own);
        ix->del_own = ix->del_rows = ix->del_slots = nullptr;
        ix->del_cap = 0;
        const size_t cap = (size_t(k) + 3) & ~size_t(3);
        RZ_CUDA_TRY(ctx, cudaMalloc(&ix->del_own, cap * 8));
        ix->del_rows = ix->del_own;
        ix->del_slots = ix->del_own + cap;
        ix->del_cap = cap;
    }
    int st = ensure_seen(ctx, size_t(n));
    if (st != RZ_OK) return st;
    st = reset_if_dirty(ctx, s);
    if (st != RZ_OK) return st;
    const uint32_t grid = grid_for(ctx, k);
    RZ_CUDA_TRY(ctx, launch_pdl(ix_claim_kernel, grid, 256, 0, s, ix->keys, ix->rows, ctx->ws.seen, ix->mask,
                                reinterpret_cast<const unsigned long long*>(d_keys), uint32_t(k), uint32_t(n),
                                ix->del_rows, ix->del_slots, ctx->ws.status));
    // The removal, unless the claims failed. The predictor reads the rows: there the host looks at the
    // outcome first.
    const bool look = (flags & RZ_USE_PREDICTOR) != 0;
    uint32_t bits = 0;
    if (look) st = fetch_status(ctx, s, &bits);
    int64_t nl = 0;
    if (st == RZ_OK && bits == 0)
        st = remove_impl(ctx, d_data, n, record_bytes, ix->del_rows, k, &nl,
                       (flags | RZ_VALIDATE | kPrevalidated) & ~uint32_t(RZ_SYNC), stream);
    // The status as the removal left it; the index update, which looks at it too, runs meanwhile.
    if (st == RZ_OK && bits == 0) st = queue_status(ctx, s);
    if (st == RZ_OK && bits == 0) {
        const cudaError_t e = launch_pdl(ix_update_kernel, grid, 256, 0, s, ix->keys, ix->rows, ctx->ws.seen, ix->mask,
                                         static_cast<const uint8_t*>(d_data), record_bytes, ix->del_rows, ix->del_slots,
                                         uint32_t(k), uint32_t(n - k), ctx->ws.status);
        st = e != cudaSuccess ? cuda_fail(ctx, e, "ix_update_kernel") : await_status(ctx, s, &bits);
    }
    if (st != RZ_OK || bits != 0) {
        // Nothing moved (or the device gave up): the index keeps its keys. The update has looked at
        // the status by the time the stream is idle.
        ix_unclaim_kernel<<<grid, 256, 0, s>>>(ctx->ws.seen, ix->del_rows, uint32_t(k), uint32_t(n));
        cudaStreamSynchronize(s);
        cudaMemset(ctx->ws.status, 0, sizeof(uint32_t));
        ctx->ws.dirty = true;
        return st != RZ_OK ? st : map_status(bits);
    }
    if (flags & RZ_SYNC) RZ_CUDA_TRY(ctx, cudaStreamSynchronize(s));
    return RZ_OK;
}

}  // extern "C"
