// rz_bulk.cu -- single-list Redzone for large k, 4-byte items: holes written line by line (the bulk
// schedule).
//
// The same rule and the same phases as the grid schedule (rz_single.cu; reference Algorithm 2,
// redzone.hxx:626-941), but a hole's item is not stored where it is found. Random stores into a list
// much larger than L2 run at about 2.2e10 per second on B200 whatever their width: each costs a
// partial-sector write of its own, and that is what the grid schedule's time goes to for large k.
// Grouping them by region is no help while a warp's stores still go to 32 different 128-byte lines
// (2^24 int32 stores into 1 GiB: 760 us in random order, 560 grouped by 4 MB, 455 by 16 KB); stores
// that share lines inside the warp instruction take 250-265 us (grouped by 1 KB, or sorted). So:
//   sample: whether the holes crowd (a list with most of its removals in the tail, or in one part), or
//          neighbours in the list lie near each other (sorted lists, runs in order). Their stores meet in
//          L2, so the grid kernel, which is launched next, does such a list. A word (gate) makes
//          either it or the four kernels behind it return at once;
//   mark:  the V map (tail positions whose item is removed; phase A's red-zone bits) and the P map
//          (entries that are no hole), and the number of holes in each of up to 2048 equal ranges of
//          the list (buckets); the last block turns the counts into bucket offsets;
//   split: entries in neither map are settled (phase B): their (hole, item) pairs go to their
//          buckets. The orphans, V \ P and P \ V, are listed in order per block; the last block turns
//          the blocks' counts into prefixes;
//   pair:  the orphans' pairs (phase C), into the same buckets, and the V map cleared for the next call;
//   fill:  a block takes bucket after bucket, orders its pairs by granules of about 1 KB in shared
//          memory and stores them in that order.
// Kernels in stream order and no wait inside any of them; one block's step of split, pair and fill is
// the same unordered counting sort in shared memory. Each hole has one pair, so the order of a
// bucket's pairs does not matter and the result is the canonical one.
//
// Which lists it is for (us per call, grid schedule / this one, lists of n int32; the last three columns' lists
// are done by the grid kernel after the sample):
//   n, k              uniform        runs of 256,    from the tail   runs in       sorted
//                                    any order                       order
//   2^28, 2^26        2510 / 1555    2307 / 1287     1300 / 1313     784 / 798     905 / 919
//   2^28, 2^24         760 /  475     414 /  328      258 /  272     166 / 180     328 / 340
//   2^28, 2^23         396 /  317     217 /  177      136 /  149      82 /  95     235 / 248
//   2^28, 3 * 2^21     312 /  270     167 /  140      109 /  121      60 /  72     205 / 219
//   2^27, 2^25        1165 /  727     855 /  667      543 /  557     407 / 421     464 / 476
//   2^27, 2^24         664 /  406     335 /  324      260 /  274     182 / 195     263 / 276
//   2^27, 3 * 2^22     522 /  330     253 /  254      193 /  206     136 / 149     207 / 217
//   2^27, 2^23         367 /  256     179 /  179      124 /  137      87 / 101     156 / 168
//   2^26, 2^24         495 /  368     242 /  344      260 /  272     213 / 227     240 / 254
//   2^26, 2^23         297 /  225     107 /  180      126 /  140      95 / 109     136 / 148
// The lists that the grid kernel does pay 10 to 14 us for the sample (3.6) and the four empty launches (2.2
// each), so the default takes it from k = 3 * 2^22, where that is 5 to 9 % and the others gain up to 1.6 times,
// and only for lists of 2^27 items or more: in shorter ones runs in any order meet in L2. Holes more than
// 64 items apart do not share lines; with fewer than three quarters of the entries holes, there is less to gain.
#include <algorithm>
#include <atomic>

#include "rz_common.cuh"
#include "rz_internal.h"

namespace rz {

constexpr uint32_t kBulkMaxBins = 2048;
constexpr uint32_t kBulkMarkLoads = 8;
constexpr int kBulkBlock = 1024;  // mark and fill
constexpr int kSplitBlock = 512;  // split and pair: two blocks per SM, one's loads beside the other's shared memory work
constexpr int kBulkIpt = 16;      // items per thread of a tile: 1024 threads' staged pairs fill one SM's shared memory

struct BulkParams {
    uint32_t* data;
    const uint32_t* idx;
    uint32_t n, k;
    uint32_t* vmap;    // k bits, zero on entry, left zero
    uint32_t* pmap;    // k bits
    uint32_t* dlist;
    uint32_t* slist;
    uint32_t* status;
    uint32_t* hist;    // kBulkMaxBins hole counts (zero on entry, left zero)
    uint32_t* done;    // blocks finished (zero on entry, left zero)
    const uint32_t* gate;  // nonzero: the grid kernel did the list
    uint32_t* ticket;  // buckets taken by the fill kernel (zero before it)
    uint32_t* base;    // kBulkMaxBins: first pair of each bucket
    uint32_t* cursor;  // kBulkMaxBins: next free pair of each bucket
    uint32_t* orph;    // 2 * (kMaxGrid + 1): destination and source orphans per block, then their prefixes
    uint2* pairs;      // k (hole, item) pairs
    uint32_t magic;    // bucket of a hole: the high word of hole * magic, which never falls as holes rise
    uint32_t nb;       // buckets
    uint32_t G, tpc;   // split blocks and tiles per block
    uint32_t validate;
};

__device__ __forceinline__ uint32_t bucket_of(const BulkParams& p, uint32_t at) { return __umulhi(at, p.magic); }

// A failed validation leaves the caller's data untouched.
__device__ __forceinline__ bool bulk_refused(const BulkParams& p) {
    return p.validate && (__ldcg(p.status) & ST_INVALID) != 0u;
}

__device__ __forceinline__ bool bulk_skip(const BulkParams& p) { return bulk_refused(p) || __ldcg(p.gate) != 0u; }

// A word that is read once: the pairs written meanwhile stay in L2 instead (without the hint the split
// takes 152 us for 2^24 entries, with it 130).
__device__ __forceinline__ uint32_t ld_l2_once(const uint32_t* a, uint64_t pol) {
    uint32_t v;
    asm volatile("ld.global.cg.L2::cache_hint.b32 %0, [%1], %2;" : "=r"(v) : "l"(a), "l"(pol));
    return v;
}

// One block's shared memory for a tile of B * kBulkIpt pairs.
template <int B>
struct SplitSmem {
    uint32_t cnt[kBulkMaxBins];   // pairs per bin, then their prefix
    uint32_t disp[kBulkMaxBins];  // (place of the bin's first pair in the output) - prefix
    uint32_t scan[33];
    uint32_t pad[3];
    uint2 stage[size_t(B) * kBulkIpt];
};

// Prefixes of the bins' counts (cnt), all threads together; returns their sum. place(bin, count) is
// called for every bin, bin q * B + t by thread t, and gives the place of the bin's first pair: all
// of a thread's places are asked for (one atomic each, in the split) before the scan, and first used
// by split_places, after the pairs were staged. Starts with a barrier; the prefixes are ready on return.
template <int B, typename Place>
__device__ __forceinline__ uint32_t split_scan(SplitSmem<B>& s, uint32_t nb, uint32_t (&at)[kBulkMaxBins / B],
                                               Place place) {
    constexpr uint32_t PER = kBulkMaxBins / B;
    __syncthreads();
#pragma unroll
    for (uint32_t q = 0; q < PER; ++q) {
        const uint32_t b = q * B + threadIdx.x;
        at[q] = place(b, b < nb ? s.cnt[b] : 0u);
    }
    uint32_t c[PER], sum = 0;
#pragma unroll
    for (uint32_t q = 0; q < PER; ++q) {
        c[q] = s.cnt[threadIdx.x * PER + q];
        sum += c[q];
    }
    uint32_t total;
    uint32_t run = block_exclusive_scan(sum, s.scan, &total);
#pragma unroll
    for (uint32_t q = 0; q < PER; ++q) {
        s.cnt[threadIdx.x * PER + q] = run;
        run += c[q];
    }
    __syncthreads();
    return total;
}

// The bins' displacements from their places; ready after the next barrier.
template <int B>
__device__ __forceinline__ void split_places(SplitSmem<B>& s, const uint32_t (&at)[kBulkMaxBins / B]) {
#pragma unroll
    for (uint32_t q = 0; q < kBulkMaxBins / B; ++q) {
        const uint32_t b = q * B + threadIdx.x;
        s.disp[b] = at[q] - s.cnt[b];
    }
}

template <int B>
__device__ __forceinline__ void split_clear(SplitSmem<B>& s) {
    for (uint32_t q = threadIdx.x; q < kBulkMaxBins; q += B) s.cnt[q] = 0u;
}

// Whether this block is the last of the grid to get here; every block's earlier writes are visible
// to it then. Resets the counter.
__device__ __forceinline__ bool last_block(uint32_t* done) {
    __shared__ uint32_t s_last;
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        s_last = atomicAdd(done, 1u) == gridDim.x - 1u ? 1u : 0u;
        if (s_last) {
            *done = 0u;
            __threadfence();
        }
    }
    __syncthreads();
    return s_last != 0u;
}

// Whether the grid kernel stores the list's holes well, from 64 rows of 32 consecutive entries (its warps'
// stores). Either the holes crowd: three eighths of the entries red or more, or an eighth or more of them
// in one of 32 equal ranges (uniform lists: 64 of 2048 in each). Or a row's holes lie together: two points
// for an entry with one of the next 8 within 1 KB of it, three more if one is in the same sector. Two
// points per entry and more are the grid kernel's (grid / bulk us, points per entry; k = 2^24 of 2^28 and
// 3 * 2^22 of 2^27): sorted 341 / 465 and 209 / 333 (2.6), sorted blocks of 8 in any order 429 / 458 and
// 282 / 324 (2.3), runs of 2 427 / 433 and 297 / 309 (2.5), of 3 325 / 412 and 253 / 304 (3.3), of 256
// 166 / 325 and 135 / 272 (4.8), four sorted lists in turn 324 / 444 and 214 / 334 (2.4); not so sorted blocks
// of 4 483 / 462 and 335 / 324 (2.0), of 2 583 / 471 and 409 / 329 (1.3), sorted with half the entries
// shuffled 621 / 475 and 418 / 338 (1.3). One block, bound by the latency of its loads.
constexpr uint32_t kCrowdSamples = 2 * kBulkBlock, kCrowdRanges = 32, kCrowdAhead = 8;
__global__ void __launch_bounds__(kBulkBlock) bulk_sample_kernel(const uint32_t* idx, uint32_t k, uint32_t cut, uint32_t* gate) {
    __shared__ uint32_t s_in[kCrowdRanges + 2];  // entries per range, red ones, points
    if (threadIdx.x < kCrowdRanges + 2) s_in[threadIdx.x] = 0u;
    const float scale = float(kCrowdRanges) / float(cut);
    const uint32_t lane = threadIdx.x & 31u, span = min(255u, cut >> 12);  // in short lists all entries are near
    pdl_begin();
    uint32_t r[2];
    bool in[2];
#pragma unroll
    for (uint32_t j = 0; j < 2; ++j) {
        const uint64_t row = (uint64_t(k) + 31u) / 32u * (j * (kBulkBlock / 32) + threadIdx.x / 32) / (kCrowdSamples / 32);
        const uint64_t i = row * 32u + lane;
        in[j] = i < k;
        r[j] = in[j] ? ld_l2(&idx[i]) : 0u;
    }
    __syncthreads();
    uint32_t points = 0;
#pragma unroll
    for (uint32_t j = 0; j < 2; ++j) {
        if (in[j]) atomicAdd(&s_in[r[j] < cut ? min(uint32_t(float(r[j]) * scale), kCrowdRanges - 1u) : kCrowdRanges], 1u);
        bool near = false, same = false;
#pragma unroll
        for (uint32_t d = 1; d <= kCrowdAhead; ++d) {
            const uint32_t o = __shfl_down_sync(0xffffffffu, r[j], d);
            const bool there = __shfl_down_sync(0xffffffffu, uint32_t(in[j]), d) != 0u && lane + d < 32u;
            near |= there && max(o, r[j]) - min(o, r[j]) <= span;
            same |= there && (o >> 3) == (r[j] >> 3);
        }
        if (in[j]) points += (near ? 2u : 0u) + (same && near ? 3u : 0u);
    }
    points = __reduce_add_sync(0xffffffffu, points);
    if (lane == 0u) atomicAdd(&s_in[kCrowdRanges + 1], points);
    __syncthreads();
    const uint32_t c = threadIdx.x <= kCrowdRanges + 1 ? s_in[threadIdx.x] : 0u;
    const uint32_t most = threadIdx.x < kCrowdRanges ? kCrowdSamples / 8u
                          : threadIdx.x == kCrowdRanges ? kCrowdSamples / 8u * 3u : kCrowdSamples * 2u;
    const bool crowd = __syncthreads_or(c >= most);
    if (threadIdx.x == 0) *gate = crowd ? 1u : 0u;
}

// Bound by the index list's read, the map's atomics and a shared-memory atomic per hole.
__global__ void __launch_bounds__(kBulkBlock, 2) bulk_mark_kernel(const BulkParams p) {
    __shared__ uint32_t s_hist[kBulkMaxBins];
    __shared__ uint32_t s_scan[33];
    for (uint32_t b = threadIdx.x; b < kBulkMaxBins; b += kBulkBlock) s_hist[b] = 0u;
    pdl_begin();
    if (bulk_skip(p)) return;
    __syncthreads();
    const uint32_t n = p.n, k = p.k, cut = n - k;
    bool oor = false;
    constexpr uint32_t U = kBulkMarkLoads;
    const uint64_t stride = uint64_t(gridDim.x) * kBulkBlock * U;
    // Whole warps: every lane of a warp runs the same number of steps (the ballot below).
    for (uint64_t b = uint64_t(blockIdx.x) * (kBulkBlock * U) + threadIdx.x; (b & ~uint64_t(31)) < k; b += stride) {
        uint32_t r[U];
#pragma unroll
        for (uint32_t j = 0; j < U; ++j) {
            const uint64_t i = b + j * uint32_t(kBulkBlock);
            r[j] = i < k ? ld_l2(&p.idx[i]) : 0u;
        }
#pragma unroll
        for (uint32_t j = 0; j < U; ++j) {
            const uint64_t i = b + j * uint32_t(kBulkBlock);
            // Rows start at multiples of 32: one word of the P map each (entries past the end count as no hole).
            const uint32_t m = __ballot_sync(0xffffffffu, i >= k || r[j] >= cut);
            if ((threadIdx.x & 31u) == 0u && i < k) p.pmap[i >> 5] = m;
            if (i >= k) continue;
            if (r[j] < cut) {
                atomicAdd(&s_hist[bucket_of(p, r[j])], 1u);
            } else if (r[j] >= n) {
                oor = true;
            } else {
                const uint32_t off = r[j] - cut;
                atomicOr(&p.vmap[off >> 5], 1u << (off & 31u));
            }
        }
    }
    if (oor) atomicOr(p.status, ST_RANGE);
    __syncthreads();
    for (uint32_t b = threadIdx.x; b < p.nb; b += kBulkBlock)
        if (s_hist[b]) atomicAdd(&p.hist[b], s_hist[b]);
    if (!last_block(p.done)) return;
    constexpr uint32_t PER = kBulkMaxBins / kBulkBlock;
    uint32_t c[PER], sum = 0;
#pragma unroll
    for (uint32_t q = 0; q < PER; ++q) {
        const uint32_t b = threadIdx.x * PER + q;
        c[q] = __ldcg(&p.hist[b]);
        p.hist[b] = 0u;
        sum += c[q];
    }
    if (threadIdx.x == 0) *p.ticket = 0u;
    uint32_t total;
    uint32_t run = block_exclusive_scan(sum, s_scan, &total);
#pragma unroll
    for (uint32_t q = 0; q < PER; ++q) {
        p.base[threadIdx.x * PER + q] = run;
        p.cursor[threadIdx.x * PER + q] = run;
        run += c[q];
    }
}

// Write a tile's staged pairs out, bucket by bucket, and clear the counts for the next tile.
__device__ __forceinline__ void bulk_write(SplitSmem<kSplitBlock>& s, const BulkParams& p, uint32_t total) {
    __syncthreads();
    split_clear(s);
#pragma unroll 4
    for (uint32_t q = threadIdx.x; q < total; q += kSplitBlock) {
        const uint2 pair = s.stage[q];
        p.pairs[s.disp[bucket_of(p, pair.x)] + q] = pair;
    }
    __syncthreads();
}

// One tile of the split: warp w owns its consecutive IPT * 32 entries, row j at +32 j.
template <bool FULL>
__device__ __forceinline__ void bulk_split_tile(SplitSmem<kSplitBlock>& s, const BulkParams& p, uint32_t base,
                                                uint32_t (&s_orph)[kSplitBlock / 32], uint32_t chunk, uint32_t& nd,
                                                uint32_t& ns) {
    constexpr int IPT = kBulkIpt;
    static_assert(IPT % 2 == 0 && IPT <= 32, "two ranks per register, one map word per lane");
    const uint32_t k = p.k, cut = p.n - k;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t wbase = base + uint32_t(warp) * (IPT * 32), i0 = wbase + lane;
    const uint32_t* idx = p.idx + i0;
    const uint32_t* tail = p.data + cut + i0;
    const uint64_t once = l2_policy_evict_first();
    uint32_t rr[IPT], rank[IPT / 2];  // entries, their 16-bit ranks in their buckets
    uint32_t src[IPT];
#pragma unroll
    for (int j = 0; j < IPT; ++j) rr[j] = FULL || i0 + j * 32 < k ? ld_l2_once(idx + j * 32, once) : 0u;
    // Lane j holds the settled entries of row j.
    uint32_t word = 0u, dst_orphans = 0u, src_orphans = 0u;
    if (lane < IPT && (FULL || wbase + uint32_t(lane) * 32u < k)) {
        const uint32_t w = (wbase >> 5) + lane;
        const uint32_t v = __ldcg(&p.vmap[w]), m = __ldcg(&p.pmap[w]);
        word = ~(v | m);
        dst_orphans = v & ~m;
        src_orphans = m & ~v;
        if (!FULL && k - wbase - uint32_t(lane) * 32u < 32u) src_orphans &= (1u << (k & 31u)) - 1u;  // P past the end
    }
    // Orphans of the tile before this lane's: destinations in the low half, sources in the high one.
    const uint32_t orphans = __popc(dst_orphans) | __popc(src_orphans) << 16;
    uint32_t before = warp_inclusive_scan(orphans);
    if (lane == 31) s_orph[warp] = before;
    before -= orphans;
    uint32_t mine = 0u;  // bit j: this lane's entry of row j is settled
#pragma unroll
    for (int j = 0; j < IPT; ++j) {
        const uint32_t set = (__shfl_sync(0xffffffffu, word, j) >> lane) & 1u;
        mine |= set << j;
        const uint32_t rk = set ? atomicAdd(&s.cnt[bucket_of(p, rr[j])], 1u) : 0u;
        if (j & 1) rank[j / 2] |= rk << 16;
        else rank[j / 2] = rk;
    }
    // The tail items arrive while the buckets' places are worked out.
#pragma unroll
    for (int j = 0; j < IPT; ++j)
        if (FULL || i0 + j * 32 < k) src[j] = ld_l2_once(tail + j * 32, once);
    uint32_t place[kBulkMaxBins / kSplitBlock];
    const uint32_t total = split_scan(s, p.nb, place, [&](uint32_t b, uint32_t c) {
        return c ? atomicAdd(&p.cursor[b], c) : 0u;
    });
    uint32_t all = 0u;
#pragma unroll
    for (int w = 0; w < kSplitBlock / 32; ++w) {
        const uint32_t x = s_orph[w];
        if (w < warp) before += x;
        all += x;
    }
    for (uint32_t at = chunk + nd + (before & 0xffffu); dst_orphans; dst_orphans &= dst_orphans - 1u)
        p.dlist[at++] = wbase + uint32_t(lane) * 32u + uint32_t(__ffs(dst_orphans) - 1);
    for (uint32_t at = chunk + ns + (before >> 16); src_orphans; src_orphans &= src_orphans - 1u)
        p.slist[at++] = wbase + uint32_t(lane) * 32u + uint32_t(__ffs(src_orphans) - 1);
    nd += all & 0xffffu;
    ns += all >> 16;
#pragma unroll
    for (int j = 0; j < IPT; ++j)
        if ((mine >> j) & 1u)
            s.stage[s.cnt[bucket_of(p, rr[j])] + ((rank[j / 2] >> (16 * (j & 1))) & 0xffffu)] = make_uint2(rr[j], src[j]);
    split_places(s, place);
    bulk_write(s, p, total);
}

__global__ void __launch_bounds__(kSplitBlock, 2) bulk_split_kernel(const BulkParams p) {
    constexpr int IPT = kBulkIpt, B = kSplitBlock, NW = B / 32;
    constexpr uint32_t TILE = uint32_t(B) * IPT;
    extern __shared__ __align__(16) uint8_t smem_raw[];
    auto& s = *reinterpret_cast<SplitSmem<B>*>(smem_raw);
    __shared__ uint32_t s_orph[NW];
    pdl_begin();
    if (bulk_skip(p)) return;
    split_clear(s);
    const uint32_t k = p.k;
    const uint32_t ntiles = (k + TILE - 1) / TILE;
    const uint32_t t0 = min(blockIdx.x * p.tpc, ntiles), t1 = min(t0 + p.tpc, ntiles);
    uint32_t nd = 0, ns = 0;
    __syncthreads();
    for (uint32_t t = t0; t < t1; ++t) {
        if (t + 1 < t1) {
            const uint32_t nb = (t + 1) * TILE, cnt = min(TILE, k - nb);
            prefetch_l2(p.idx + nb, size_t(cnt) * 4);
            prefetch_l2(p.data + (uint64_t(p.n - k) + nb), size_t(cnt) * 4);
        }
        if (k - t * TILE >= TILE) bulk_split_tile<true>(s, p, t * TILE, s_orph, t0 * TILE, nd, ns);
        else bulk_split_tile<false>(s, p, t * TILE, s_orph, t0 * TILE, nd, ns);
    }
    const uint32_t G = p.G;
    if (threadIdx.x == 0) {
        p.orph[blockIdx.x] = nd;
        p.orph[G + 1 + blockIdx.x] = ns;
    }
    if (!last_block(p.done)) return;
    uint32_t* pd = reinterpret_cast<uint32_t*>(s.stage);  // the staging area is free now
    uint32_t* ps = pd + G + 1;
    for (uint32_t c = threadIdx.x; c < G; c += B) {
        pd[c] = __ldcg(&p.orph[c]);
        ps[c] = __ldcg(&p.orph[G + 1 + c]);
    }
    __syncthreads();
    block_scan_array(pd, int(G), s.scan);
    block_scan_array(ps, int(G), s.scan);
    for (uint32_t c = threadIdx.x; c <= G; c += B) {
        p.orph[c] = pd[c];
        p.orph[G + 1 + c] = ps[c];
    }
    if (threadIdx.x == 0 && pd[G] != ps[G]) atomicOr(p.status, ST_INCONSISTENT);
}

// Bound by the gathers of the orphans' holes and items.
__global__ void __launch_bounds__(kSplitBlock, 2) bulk_pair_kernel(const BulkParams p) {
    constexpr int IPT = kBulkIpt, B = kSplitBlock;
    constexpr uint32_t TILE = uint32_t(B) * IPT;
    extern __shared__ __align__(16) uint8_t smem_raw[];
    auto& s = *reinterpret_cast<SplitSmem<B>*>(smem_raw);
    __shared__ uint32_t s_pd[kMaxGrid + 1], s_ps[kMaxGrid + 1];
    pdl_begin();
    if (bulk_skip(p)) return;
    split_clear(s);
    const uint32_t G = p.G;
    for (uint32_t c = threadIdx.x; c <= G; c += B) {
        s_pd[c] = __ldcg(&p.orph[c]);
        s_ps[c] = __ldcg(&p.orph[G + 1 + c]);
    }
    for (uint32_t q = blockIdx.x * B + threadIdx.x; q < (p.k + 31u) / 32u; q += gridDim.x * B) p.vmap[q] = 0u;
    __syncthreads();
    const uint32_t m = min(s_pd[G], s_ps[G]);  // pairs
    // A share of the pairs for every block, at most a tile at a time.
    const uint32_t share = (m + gridDim.x - 1) / gridDim.x;
    const uint32_t lo = min(blockIdx.x * share, m), hi = min(lo + share, m);
    if (lo >= hi) return;
    const uint32_t* tail = p.data + (p.n - p.k);
    const uint32_t chunk = p.tpc * TILE;  // entries of a split block, and its places in the orphan lists
    for (uint32_t base = lo; base < hi; base += TILE) {
        uint32_t at[IPT], rank[IPT / 2];
        uint32_t v[IPT];
#pragma unroll
        for (int j = 0; j < IPT; ++j) {
            const uint32_t r = base + uint32_t(j) * B + threadIdx.x;
            at[j] = 0u;
            if (r < hi) {
                const uint32_t c = owner_of_rank(s_pd, int(G), r);
                at[j] = __ldcg(&p.dlist[size_t(c) * chunk + (r - s_pd[c])]);
            }
            rank[j / 2] = 0u;
        }
#pragma unroll
        for (int j = 0; j < IPT; ++j)
            if (base + uint32_t(j) * B + threadIdx.x < hi) at[j] = ld_l2(&p.idx[at[j]]);
#pragma unroll
        for (int j = 0; j < IPT; ++j) {
            const uint32_t r = base + uint32_t(j) * B + threadIdx.x;
            const uint32_t rk = r < hi ? atomicAdd(&s.cnt[bucket_of(p, at[j])], 1u) : 0u;
            if (j & 1) rank[j / 2] |= rk << 16;
            else rank[j / 2] = rk;
            if (r < hi) {
                const uint32_t c = owner_of_rank(s_ps, int(G), r);
                v[j] = ld_l2(&tail[__ldcg(&p.slist[size_t(c) * chunk + (r - s_ps[c])])]);
            }
        }
        uint32_t place[kBulkMaxBins / kSplitBlock];
        const uint32_t total = split_scan(s, p.nb, place, [&](uint32_t b, uint32_t c) {
            return c ? atomicAdd(&p.cursor[b], c) : 0u;
        });
#pragma unroll
        for (int j = 0; j < IPT; ++j)
            if (base + uint32_t(j) * B + threadIdx.x < hi)
                s.stage[s.cnt[bucket_of(p, at[j])] + ((rank[j / 2] >> (16 * (j & 1))) & 0xffffu)] = make_uint2(at[j], v[j]);
        split_places(s, place);
        bulk_write(s, p, total);
    }
}

// Bound by the stores' partial-sector writes. A bucket's pairs (one tile of them, unless holes are
// dense) are ordered by granules of 1/1024 to 1/2048 of the bucket's range: about 1 KB where holes are
// so far apart that order pays, and finer where they are denser.
__global__ void __launch_bounds__(kBulkBlock, 1) bulk_fill_kernel(const BulkParams p) {
    constexpr int IPT = kBulkIpt, B = kBulkBlock, U = 4;
    constexpr uint32_t TILE = uint32_t(B) * IPT;
    extern __shared__ __align__(16) uint8_t smem_raw[];
    auto& s = *reinterpret_cast<SplitSmem<B>*>(smem_raw);
    __shared__ uint32_t s_next;
    pdl_begin();
    if (bulk_skip(p)) return;
    split_clear(s);
    auto first = [&](uint32_t x) {  // the lowest position of bucket x
        return uint32_t(min(((uint64_t(x) << 32) + p.magic - 1u) / p.magic, uint64_t(p.n - p.k)));
    };
    // The next bucket by a counter (the blocks' shares of the memory differ; in turn: 10 us more at 2^24).
    for (uint32_t b = blockIdx.x; b < p.nb; b = s_next) {
        __syncthreads();  // s_next was read, the bins are clear
        if (threadIdx.x == 0) s_next = gridDim.x + atomicAdd(p.ticket, 1u);
        const uint32_t start = first(b), range = first(b + 1u) - start;
        uint32_t shift = 0;
        while ((range >> shift) > kBulkMaxBins - 1) ++shift;
        const uint32_t lo = __ldcg(&p.base[b]), hi = __ldcg(&p.cursor[b]);  // up to cursor: invalid lists may lack orphans
        for (uint32_t base = lo; base < hi; base += TILE) {
            uint32_t rank[IPT / 2];
#pragma unroll
            for (int j0 = 0; j0 < IPT; j0 += U) {
                uint32_t at[U];
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const uint32_t e = base + uint32_t(j0 + u) * B + threadIdx.x;
                    at[u] = e < hi ? __ldcg(&p.pairs[e].x) : 0u;
                }
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const int j = j0 + u;
                    const bool in = base + uint32_t(j) * B + threadIdx.x < hi;
                    const uint32_t rk = in ? atomicAdd(&s.cnt[(at[u] - start) >> shift], 1u) : 0u;
                    if (j & 1) rank[j / 2] |= rk << 16;
                    else rank[j / 2] = rk;
                }
            }
            uint32_t none[kBulkMaxBins / kBulkBlock];
            const uint32_t total = split_scan(s, kBulkMaxBins, none, [](uint32_t, uint32_t) { return 0u; });
#pragma unroll
            for (int j0 = 0; j0 < IPT; j0 += U) {
                uint2 pair[U];
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const uint32_t e = base + uint32_t(j0 + u) * B + threadIdx.x;
                    if (e < hi) pair[u] = __ldcg(&p.pairs[e]);
                }
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const int j = j0 + u;
                    if (base + uint32_t(j) * B + threadIdx.x < hi)
                        s.stage[s.cnt[(pair[u].x - start) >> shift] + ((rank[j / 2] >> (16 * (j & 1))) & 0xffffu)] = pair[u];
                }
            }
            __syncthreads();
            split_clear(s);
            for (uint32_t q = threadIdx.x; q < total; q += B) p.data[s.stage[q].x] = s.stage[q].y;
            __syncthreads();
        }
        __syncthreads();
    }
}

// ------------------------------------------------------------------------------------------------
// Host side
// ------------------------------------------------------------------------------------------------
bool bulk_wanted(uint32_t n, uint32_t k, uint32_t w) {
    return w == 4 && k >= kBulkMinK && n >= kBulkMinN && n / 64u <= k && n / 4u >= k;
}

size_t bulk_counter_words() { return 3 * size_t(kBulkMaxBins) + 32 + 2 * (size_t(kMaxGrid) + 1); }

int launch_bulk_sample(rz_ctx* ctx, uint32_t n, const uint32_t* idx, uint32_t k, cudaStream_t s) {
    RZ_CUDA_TRY(ctx, launch_pdl(bulk_sample_kernel, 1, kBulkBlock, 0, s, idx, k, n - k, ctx->ws.bulk_ctr));
    return RZ_OK;
}

int launch_bulk(rz_ctx* ctx, void* data, uint32_t n, const uint32_t* idx, uint32_t k, bool validate, cudaStream_t s) {
    const uint32_t cut = n - k;
    const int smem_fill = int(sizeof(SplitSmem<kBulkBlock>)), smem_split = int(sizeof(SplitSmem<kSplitBlock>));
    static std::atomic<uint64_t> attr_set{0};
    const uint64_t dev_bit = 1ull << (ctx->device & 63);
    if (!(attr_set.load() & dev_bit)) {
        const auto dyn = cudaFuncAttributeMaxDynamicSharedMemorySize;
        RZ_CUDA_TRY(ctx, cudaFuncSetAttribute((const void*)bulk_split_kernel, dyn, smem_split));
        RZ_CUDA_TRY(ctx, cudaFuncSetAttribute((const void*)bulk_pair_kernel, dyn, smem_split));
        RZ_CUDA_TRY(ctx, cudaFuncSetAttribute((const void*)bulk_fill_kernel, dyn, smem_fill));
        attr_set.fetch_or(dev_bit);
    }
    BulkParams p{};
    p.data = static_cast<uint32_t*>(data);
    p.idx = idx;
    p.n = n;
    p.k = k;
    p.vmap = ctx->ws.bitmap;
    p.pmap = ctx->ws.bulk_pmap;
    p.dlist = ctx->ws.dlist;
    p.slist = ctx->ws.slist;
    p.status = ctx->ws.status;
    p.gate = ctx->ws.bulk_ctr;
    p.done = ctx->ws.bulk_ctr + 1;
    p.ticket = ctx->ws.bulk_ctr + 2;
    p.hist = ctx->ws.bulk_ctr + 32;
    p.base = p.hist + kBulkMaxBins;
    p.cursor = p.base + kBulkMaxBins;
    p.orph = p.cursor + kBulkMaxBins;
    p.pairs = ctx->ws.bulk_pairs;
    // Buckets of three quarters of a fill tile, so that one with a third more holes than the rest is
    // still one tile.
    constexpr uint32_t FILL = uint32_t(kBulkBlock) * kBulkIpt, TILE = uint32_t(kSplitBlock) * kBulkIpt;
    const uint64_t holes = uint64_t(k) * cut / n;
    const uint32_t want = uint32_t(std::min<uint64_t>(std::min<uint64_t>(holes / (FILL / 4 * 3) + 1, kBulkMaxBins), cut));
    p.magic = uint32_t(std::min<uint64_t>((uint64_t(want) << 32) / cut, 0xffffffffu));
    p.nb = uint32_t((uint64_t(cut - 1u) * p.magic) >> 32) + 1u;
    p.validate = validate ? 1u : 0u;
    const uint32_t ntiles = (k + TILE - 1) / TILE, g = std::min<uint32_t>(ntiles, 2u * uint32_t(ctx->sms));
    p.tpc = (ntiles + g - 1) / g;
    p.G = (ntiles + p.tpc - 1) / p.tpc;
    RZ_CUDA_TRY(ctx, launch_pdl(bulk_mark_kernel, 2 * ctx->sms, kBulkBlock, 0, s, p));
    RZ_CUDA_TRY(ctx, injected_failure(ctx));
    RZ_CUDA_TRY(ctx, launch_pdl(bulk_split_kernel, p.G, kSplitBlock, smem_split, s, p));
    RZ_CUDA_TRY(ctx, injected_failure(ctx));
    RZ_CUDA_TRY(ctx, launch_pdl(bulk_pair_kernel, 2 * ctx->sms, kSplitBlock, smem_split, s, p));
    RZ_CUDA_TRY(ctx, injected_failure(ctx));
    RZ_CUDA_TRY(ctx, launch_pdl(bulk_fill_kernel, std::min<uint32_t>(p.nb, ctx->sms), kBulkBlock, smem_fill, s, p));
    return RZ_OK;
}

}  // namespace rz
