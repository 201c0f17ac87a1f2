// Particle cell-sort: key = (tile, bin in tile) of the particle's stencil
// start, then a stable LSD radix sort of (key, particle index) pairs, then
// per-tile particle offsets.  Also the member gather used to apply the
// permutation to particle storage.
//
// Radix pass (digit width <= 9 bits), three launches:
//   * the digits of every block of elements are counted (for the first pass in
//     the kernel that computes the keys) into a digit-major table;
//   * one CTA per digit turns its row of the table into offsets among that
//     digit's elements;
//   * every block ranks its elements among equal digits in original order (the
//     lanes with the same digit from one ballot per digit bit, a running count
//     per warp, a prefix over the block's warps: stable), puts them in digit
//     order in shared memory and writes them from there, so that the elements of
//     a digit leave as one run.
// Bound: the latency of a block's phases (load, rank, write) at 32 warps per SM;
// the 16 bytes per element and pass would take 41 us of the 144.  16.8 M
// clustered particles in random order: 1.02 ms with a digit table of 2048-element
// blocks, elements written straight from their lanes and a three-launch scan of
// the table, 0.66 ms now; nearly sorted (a time loop) 0.70 -> 0.66 ms.
// Up to kSmallSort particles are sorted by a single CTA in one launch, tile
// offsets and work items included: such a sort costs launches, not bandwidth
// (6912 particles: 16 launches, 42 us on the device -> 1 launch, 21 us).
#include <cmath>

#include "binkey.cuh"

namespace pb {

constexpr int kMaxDigitBits = 9;
constexpr int kDigits = 1 << kMaxDigitBits;
constexpr int kSortThreads = 256;
constexpr int kSortWarps = kSortThreads / 32;
// Elements per thread of a block.  12: the elements of a digit leave a block in
// runs of 12 of random keys (8 bits), 4 CTAs per SM (16.8 M particles, a pass:
// 144 us; 16 elements 151, 24 with 3 CTAs 228, 512 threads with 8 / 12 / 16
// elements 156 / 160 / 167); 8 where 12 would leave SMs without a block.
constexpr int kSortItems = 12, kSortItemsFew = 8;
constexpr int kSmallSort = 8192;
constexpr int kSmallThreads = 1024, kSmallItems = kSmallSort / kSmallThreads;
constexpr int64_t kSmallTiles = 16384;  // tiles a single CTA still handles well
constexpr int kScanThreads = 1024;
constexpr int kScanItems = 4;
constexpr int kScanTile = kScanThreads * kScanItems;

// Lanes of the warp whose digit (of at most BITS bits) equals this lane's, among
// the lanes with the same `valid`.
template <int BITS>
__device__ __forceinline__ unsigned equal_digits(uint32_t dig, bool valid)
{
    const unsigned vm = __ballot_sync(0xFFFFFFFFu, valid);
    unsigned peers = valid ? vm : ~vm;
#pragma unroll
    for (int b = 0; b < BITS; ++b) {
        const bool bit = (dig >> b) & 1u;
        const unsigned m = __ballot_sync(0xFFFFFFFFu, bit);
        peers &= bit ? m : ~m;
    }
    return peers;
}

// Counts a warp's digits into shared counters; a warp whose digits are all the
// same (nearly sorted keys) adds once.
__device__ __forceinline__ void count_digits(uint32_t* cnt, uint32_t dig, bool valid)
{
    const unsigned vm = __ballot_sync(0xFFFFFFFFu, valid);
    if (!vm) return;
    const uint32_t first = __shfl_sync(0xFFFFFFFFu, dig, __ffs(vm) - 1);
    if (__all_sync(0xFFFFFFFFu, !valid || dig == first)) {
        if ((threadIdx.x & 31) == 0) atomicAdd(&cnt[first], (uint32_t)__popc(vm));
    } else if (valid) {
        atomicAdd(&cnt[dig], 1u);
    }
}

// Digit counts of block blockIdx.x of the elements into column blockIdx.x of
// the digit-major table.  KEYS: the keys are computed from the positions and
// written first.
template <int ITEMS, bool KEYS>
__global__ void __launch_bounds__(kSortThreads)
radix_count_kernel(BinP bp, PField x, const uint32_t* __restrict__ kin, uint32_t* __restrict__ kout,
                   int64_t n, int shift, int bits, uint32_t* __restrict__ table, int64_t nblk,
                   uint32_t kmax)
{
    __shared__ uint32_t cnt[kDigits];
    const int nd = 1 << bits;
    const uint32_t mask = (uint32_t)nd - 1;
    for (int i = threadIdx.x; i < nd; i += kSortThreads) cnt[i] = 0;
    __syncthreads();
    const int64_t base = (int64_t)blockIdx.x * (kSortThreads * ITEMS) + threadIdx.x;
#pragma unroll(KEYS ? 4 : ITEMS)
    for (int r = 0; r < ITEMS; ++r) {
        const int64_t e = base + r * kSortThreads;
        const bool valid = e < n;
        uint32_t key = 0;
        if constexpr (KEYS) {
            if (valid) {
                const double xs[3] = {x.get<double>(e, 0), x.get<double>(e, 1), x.get<double>(e, 2)};
                key = particle_key(bp, xs);
                kout[e] = key;
            }
        } else {
            key = valid ? min(__ldg(kin + e), kmax) : 0u;
        }
        count_digits(cnt, (key >> shift) & mask, valid);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < nd; i += kSortThreads) table[(int64_t)i * nblk + blockIdx.x] = cnt[i];
}

// Exclusive prefix of v over the CTA's threads (warp_sums: 32 words).
__device__ __forceinline__ uint32_t block_exclusive_scan(uint32_t v, uint32_t* warp_sums,
                                                         uint32_t* total)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t inc = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(0xFFFFFFFFu, inc, o);
        if (lane >= o) inc += t;
    }
    if (lane == 31) warp_sums[warp] = inc;
    __syncthreads();
    if (warp == 0) {
        const int nw = blockDim.x >> 5;
        uint32_t s = lane < nw ? warp_sums[lane] : 0u;
        uint32_t si = s;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t t = __shfl_up_sync(0xFFFFFFFFu, si, o);
            if (lane >= o) si += t;
        }
        if (lane < nw) warp_sums[lane] = si - s;
        if (lane == 31) *total = si;
    }
    __syncthreads();
    const uint32_t r = warp_sums[warp] + inc - v;
    __syncthreads();
    return r;
}

// Row blockIdx.x of the table: counts -> exclusive prefix; its sum to totals.
__global__ void __launch_bounds__(kSortThreads)
radix_row_kernel(uint32_t* __restrict__ table, int64_t nblk, uint32_t* __restrict__ totals)
{
    __shared__ uint32_t ws[32];
    __shared__ uint32_t total;
    uint32_t* row = table + (int64_t)blockIdx.x * nblk;
    uint32_t carry = 0;
    for (int64_t base = 0; base < nblk; base += kSortThreads * 4) {
        uint32_t v[4], sum = 0;
        const int64_t e = base + (int64_t)threadIdx.x * 4;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            v[q] = e + q < nblk ? row[e + q] : 0u;
            sum += v[q];
        }
        uint32_t run = carry + block_exclusive_scan(sum, ws, &total);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            if (e + q < nblk) row[e + q] = run;
            run += v[q];
        }
        carry += total;
        __syncthreads();
    }
    if (threadIdx.x == 0) totals[blockIdx.x] = carry;
}

// Shared memory of a block that ranks TILE elements with WARPS warps.
template <int TILE, int WARPS, int DIGITS>
struct RankSmem {
    uint32_t key[TILE], val[TILE];
    uint32_t cnt[WARPS][DIGITS];  // per warp: counts, then offsets among its digit
    uint32_t start[DIGITS];       // first element of a digit in the block's order
    uint32_t ws[32];
    uint32_t total;
};

// Ranks the block's elements (warp-striped: item r of lane l of warp w is element
// (w ITEMS + r) 32 + l) by digit, stable, and puts them in that order into
// S.key / S.val.  Called by all THREADS (>= DIGITS) threads; S.start and S.cnt are
// left for the caller, who syncs before reading S.
template <int THREADS, int ITEMS, int BITS, class S>
__device__ __forceinline__ void rank_block(S& sm, const uint32_t (&key)[ITEMS],
                                           const uint32_t (&val)[ITEMS], int live, int shift, int bits)
{
    constexpr int PER = (1 << BITS) > THREADS ? (1 << BITS) / THREADS : 1;  // digits per thread
    const int nd = 1 << bits;
    const uint32_t mask = (uint32_t)nd - 1;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int i = lane; i < nd; i += 32) sm.cnt[warp][i] = 0;
    __syncwarp();
    const unsigned below = (1u << lane) - 1u;
    // The last lane of every digit adds the digit's count to the warp's counter;
    // what it was before is the digit's count in the items before (the adds of
    // successive items are in order, and in flight together).
    uint32_t rank[ITEMS];
#pragma unroll
    for (int r = 0; r < ITEMS; ++r) {
        const bool valid = (warp * ITEMS + r) * 32 + lane < live;
        const uint32_t dig = (key[r] >> shift) & mask;
        const unsigned peers = equal_digits<BITS>(dig, valid);
        const int last = 31 - __clz(peers);
        uint32_t before = 0;
        if (valid && lane == last) before = atomicAdd(&sm.cnt[warp][dig], (uint32_t)__popc(peers));
        __syncwarp();
        rank[r] = __shfl_sync(0xFFFFFFFFu, before, last) + (uint32_t)__popc(peers & below);
    }
    __syncthreads();
    uint32_t count[PER], sum = 0;
#pragma unroll
    for (int q = 0; q < PER; ++q) {
        const int d = (int)threadIdx.x * PER + q;
        count[q] = 0;
        if (d < nd) {
#pragma unroll 8
            for (int w = 0; w < THREADS / 32; ++w) {
                const uint32_t t = sm.cnt[w][d];
                sm.cnt[w][d] = count[q];
                count[q] += t;
            }
        }
        sum += count[q];
    }
    uint32_t first = block_exclusive_scan(sum, sm.ws, &sm.total);
#pragma unroll
    for (int q = 0; q < PER; ++q) {
        const int d = (int)threadIdx.x * PER + q;
        if (d < nd) sm.start[d] = first;
        first += count[q];
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < ITEMS; ++r) {
        if ((warp * ITEMS + r) * 32 + lane < live) {
            const uint32_t dig = (key[r] >> shift) & mask;
            const uint32_t pos = sm.start[dig] + sm.cnt[warp][dig] + rank[r];
            sm.key[pos] = key[r];
            sm.val[pos] = val[r];
        }
    }
}

template <int ITEMS, int BITS>
using ScatterSmem = RankSmem<kSortThreads * ITEMS, kSortWarps, (1 << BITS)>;

// Block blockIdx.x of the elements to its places in kout / vout.  vin null: an
// element's value is its index.
template <int ITEMS, int BITS>
__global__ void __launch_bounds__(kSortThreads, 4)
radix_scatter_kernel(const uint32_t* __restrict__ kin, const uint32_t* __restrict__ vin,
                     uint32_t* __restrict__ kout, uint32_t* __restrict__ vout, int64_t n, int shift,
                     int bits, const uint32_t* __restrict__ table,
                     const uint32_t* __restrict__ totals, int64_t nblk, uint32_t kmax)
{
    extern __shared__ __align__(16) unsigned char sort_smem[];
    using Smem = ScatterSmem<ITEMS, BITS>;
    Smem& sm = *reinterpret_cast<Smem*>(sort_smem);
    const int nd = 1 << bits;
    const uint32_t mask = (uint32_t)nd - 1;
    const int64_t base = (int64_t)blockIdx.x * (kSortThreads * ITEMS);
    const int live = (int)min((int64_t)(kSortThreads * ITEMS), n - base);
    const int e0 = (threadIdx.x >> 5) * 32 * ITEMS + (threadIdx.x & 31);
    uint32_t key[ITEMS], val[ITEMS];
#pragma unroll
    for (int r = 0; r < ITEMS; ++r) {
        const bool valid = e0 + 32 * r < live;
        key[r] = valid ? min(__ldg(kin + base + e0 + 32 * r), kmax) : 0u;
        val[r] = !valid ? 0u : (vin ? __ldg(vin + base + e0 + 32 * r) : (uint32_t)(base + e0 + 32 * r));
    }
    // first place of this block's elements of a digit
    constexpr int PER = (1 << BITS) > kSortThreads ? (1 << BITS) / kSortThreads : 1;
    uint32_t place[PER], sum = 0;
#pragma unroll
    for (int q = 0; q < PER; ++q) {
        const int d = (int)threadIdx.x * PER + q;
        place[q] = d < nd ? totals[d] : 0u;
        sum += place[q];
    }
    uint32_t run = block_exclusive_scan(sum, sm.ws, &sm.total);
#pragma unroll
    for (int q = 0; q < PER; ++q) {
        const int d = (int)threadIdx.x * PER + q;
        const uint32_t t = place[q];
        place[q] = d < nd ? run + table[(int64_t)d * nblk + blockIdx.x] : 0u;
        run += t;
    }
    rank_block<kSortThreads, ITEMS, BITS>(sm, key, val, live, shift, bits);
    __syncthreads();
    // element i of the block's order goes to place[digit] + i - start[digit]
    uint32_t* offset = sm.cnt[0];  // (the counts are done with)
#pragma unroll
    for (int q = 0; q < PER; ++q) {
        const int d = (int)threadIdx.x * PER + q;
        if (d < nd) offset[d] = place[q] - sm.start[d];
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < ITEMS; ++r) {
        const int i = threadIdx.x + r * kSortThreads;
        if (i < live) {
            const uint32_t k = sm.key[i];
            const uint32_t pos = offset[(k >> shift) & mask] + (uint32_t)i;
            kout[pos] = k;
            vout[pos] = sm.val[i];
        }
    }
}

// First element of the sorted keys (count n) that is not below `target`.
__device__ __forceinline__ int64_t lower_bound(const uint32_t* keys, int64_t n, uint64_t target)
{
    int64_t lo = 0, hi = n;
    while (lo < hi) {
        const int64_t mid = (lo + hi) >> 1;
        if ((uint64_t)keys[mid] < target) lo = mid + 1;
        else hi = mid;
    }
    return lo;
}

// The whole sort of n <= kSmallSort particles by one CTA: keys from the
// positions (key_src null) or from the caller's keys, radix passes of 8 bits in
// shared memory, tile offsets and the work-item prefix.
using SmallSmem = RankSmem<kSmallSort, kSmallThreads / 32, 256>;

__global__ void __launch_bounds__(kSmallThreads)
small_sort_kernel(BinP bp, int n, PField x, const uint32_t* __restrict__ key_src, int nbits,
                  uint32_t* __restrict__ key_out, uint32_t* __restrict__ perm, int64_t ntiles,
                  int chunk, int64_t* __restrict__ tile_offset, uint32_t* __restrict__ tile_items)
{
    extern __shared__ __align__(16) unsigned char sort_smem[];
    SmallSmem& sm = *reinterpret_cast<SmallSmem*>(sort_smem);
    const int e0 = (threadIdx.x >> 5) * 32 * kSmallItems + (threadIdx.x & 31);
    uint32_t key[kSmallItems], val[kSmallItems];
#pragma unroll
    for (int r = 0; r < kSmallItems; ++r) {
        const int e = e0 + 32 * r;
        key[r] = 0u;
        val[r] = (uint32_t)e;
        if (e < n) {
            if (key_src) {
                key[r] = min(__ldg(key_src + e), bp.nkeys);
            } else {
                const double xs[3] = {x.get<double>(e, 0), x.get<double>(e, 1), x.get<double>(e, 2)};
                key[r] = particle_key(bp, xs);
            }
        }
    }
    for (int shift = 0; shift < nbits; shift += 8) {
        const int bits = min(8, nbits - shift);
        rank_block<kSmallThreads, kSmallItems, 8>(sm, key, val, n, shift, bits);
        __syncthreads();
#pragma unroll
        for (int r = 0; r < kSmallItems; ++r) {
            const int e = e0 + 32 * r;
            if (e < n) {
                key[r] = sm.key[e];
                val[r] = sm.val[e];
            }
        }
        __syncthreads();  // (read before the next pass writes)
    }
#pragma unroll
    for (int r = 0; r < kSmallItems; ++r) {
        const int e = e0 + 32 * r;
        if (e < n) {
            key_out[e] = key[r];
            perm[e] = val[r];
        }
    }
    uint32_t carry = 0;
    for (int64_t base = 0; base <= ntiles; base += kSmallThreads) {
        const int64_t t = base + threadIdx.x;
        uint32_t items = 0;
        if (t <= ntiles) {
            const int64_t lo = lower_bound(sm.key, n, (uint64_t)t * bp.tsize);
            tile_offset[t] = lo;
            if (t < ntiles) {
                const int64_t cnt = lower_bound(sm.key, n, (uint64_t)(t + 1) * bp.tsize) - lo;
                items = (uint32_t)((cnt + chunk - 1) / chunk);
            }
        }
        const uint32_t ex = block_exclusive_scan(items, sm.ws, &sm.total);
        if (t <= ntiles) tile_items[t] = carry + ex;
        carry += sm.total;
        __syncthreads();
    }
}

// ---------------------------------------------------------------------------
// exclusive scan of a uint32 array (three phases)
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(kScanThreads)
scan_reduce_kernel(const uint32_t* __restrict__ in, int64_t m, uint32_t* __restrict__ sums)
{
    __shared__ uint32_t red[kScanThreads / 32];
    const int64_t base = (int64_t)blockIdx.x * kScanTile + (int64_t)threadIdx.x * kScanItems;
    uint32_t s = 0;
#pragma unroll
    for (int q = 0; q < kScanItems; ++q)
        if (base + q < m) s += in[base + q];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xFFFFFFFFu, s, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x < 32) {
        uint32_t t = red[threadIdx.x];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) t += __shfl_down_sync(0xFFFFFFFFu, t, o);
        if (threadIdx.x == 0) sums[blockIdx.x] = t;
    }
}

// Single block: exclusive scan of the block sums in place.
__global__ void __launch_bounds__(kScanThreads) scan_sums_kernel(uint32_t* sums, int64_t nb)
{
    __shared__ uint32_t ws[32];
    __shared__ uint32_t total;
    uint32_t carry = 0;
    for (int64_t base = 0; base < nb; base += kScanThreads) {
        const int64_t e = base + threadIdx.x;
        const uint32_t v = e < nb ? sums[e] : 0u;
        const uint32_t ex = block_exclusive_scan(v, ws, &total);
        if (e < nb) sums[e] = carry + ex;
        carry += total;
        __syncthreads();
    }
}

__global__ void __launch_bounds__(kScanThreads)
scan_apply_kernel(const uint32_t* __restrict__ in, uint32_t* __restrict__ out, int64_t m,
                  const uint32_t* __restrict__ sums)
{
    __shared__ uint32_t ws[32];
    __shared__ uint32_t total;
    const int64_t base = (int64_t)blockIdx.x * kScanTile + (int64_t)threadIdx.x * kScanItems;
    uint32_t v[kScanItems];
    uint32_t s = 0;
#pragma unroll
    for (int q = 0; q < kScanItems; ++q) {
        v[q] = (base + q < m) ? in[base + q] : 0u;
        s += v[q];
    }
    uint32_t run = block_exclusive_scan(s, ws, &total) + sums[blockIdx.x];
#pragma unroll
    for (int q = 0; q < kScanItems; ++q) {
        if (base + q < m) out[base + q] = run;
        run += v[q];
    }
}

// Per tile: first particle, and the number of its work items (warps of 31 tiles
// and the next warp's first one, so that every offset is searched once).
__global__ void tile_offset_kernel(const uint32_t* __restrict__ keys, int64_t n, int64_t ntiles,
                                   uint32_t tsize, int chunk, int64_t* __restrict__ tile_offset,
                                   uint32_t* __restrict__ items)
{
    const int lane = threadIdx.x & 31;
    const int64_t warps = (int64_t)gridDim.x * blockDim.x / 32;
    for (int64_t w = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) / 32; w * 31 <= ntiles; w += warps) {
        const int64_t t = w * 31 + lane;
        const int64_t lo = t <= ntiles ? lower_bound(keys, n, (uint64_t)t * tsize) : n;
        const int64_t next = __shfl_down_sync(0xFFFFFFFFu, lo, 1);
        if (lane < 31 && t <= ntiles) {
            tile_offset[t] = lo;
            items[t] = t < ntiles ? (uint32_t)((next - lo + chunk - 1) / chunk) : 0u;
        }
    }
}

// Exclusive prefix of m <= kSmallTiles + 1 counts by one CTA.
__global__ void __launch_bounds__(kScanThreads)
scan_one_kernel(const uint32_t* __restrict__ in, uint32_t* __restrict__ out, int m)
{
    __shared__ uint32_t ws[32];
    __shared__ uint32_t total;
    uint32_t carry = 0;
    for (int base = 0; base < m; base += kScanTile) {
        const int e = base + (int)threadIdx.x * kScanItems;
        uint32_t v[kScanItems], sum = 0;
#pragma unroll
        for (int q = 0; q < kScanItems; ++q) {
            v[q] = e + q < m ? in[e + q] : 0u;
            sum += v[q];
        }
        uint32_t run = carry + block_exclusive_scan(sum, ws, &total);
#pragma unroll
        for (int q = 0; q < kScanItems; ++q) {
            if (e + q < m) out[e + q] = run;
            run += v[q];
        }
        carry += total;
        __syncthreads();
    }
}

template <class T>
__global__ void permute_kernel(int64_t n, int ncomp, const uint32_t* __restrict__ perm, PField src,
                               PField dst)
{
    for (int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; p < n;
         p += (int64_t)gridDim.x * blockDim.x) {
        const int64_t q = perm[p];
        for (int c = 0; c < ncomp; ++c) dst.set<T>(p, c, src.get<T>(q, c));
    }
}

// Packed rows (array of structures): one thread per (particle, word) with the
// widest word that divides the row and both base addresses, so that the
// stores of a warp are contiguous and a row is read in whole words; four
// elements per thread, their gathers in flight together.  WORDS > 0: the words
// of a row as a constant (the division by it was half of the instructions).
// 16.8 M nearly sorted particles: 48-byte rows 301 -> 263 us, 24-byte rows 219 ->
// 178 us, 4-byte rows 73 -> 36 us; in random order (bound by the 64-byte DRAM
// reads of single rows) 546 -> 527, 423 -> 398, 97 -> 84 us.
constexpr int kPermuteItems = 4;

template <class W, int WORDS>
__global__ void __launch_bounds__(256)
permute_rows_kernel(int64_t n, int words_rt, const uint32_t* __restrict__ perm,
                    const W* __restrict__ src, W* __restrict__ dst)
{
    const int words = WORDS > 0 ? WORDS : words_rt;
    const int64_t total = n * words;
    const int64_t e0 = (int64_t)blockIdx.x * (256 * kPermuteItems) + threadIdx.x;
    W v[kPermuteItems];
#pragma unroll
    for (int q = 0; q < kPermuteItems; ++q) {
        const int64_t e = e0 + q * 256;
        if (e < total) {
            const int64_t p = WORDS > 0 ? e / WORDS : e / words;
            v[q] = __ldg(src + (int64_t)__ldg(perm + p) * words + (int)(e - p * words));
        }
    }
#pragma unroll
    for (int q = 0; q < kPermuteItems; ++q)
        if (e0 + q * 256 < total) dst[e0 + q * 256] = v[q];
}

template <class W>
static void launch_permute_rows(int64_t n, int words, const uint32_t* perm, const void* src,
                                void* dst, cudaStream_t s)
{
    const unsigned blocks = (unsigned)((n * words + 256 * kPermuteItems - 1) / (256 * kPermuteItems));
    auto launch = [&](auto kern) {
        kern<<<blocks, 256, 0, s>>>(n, words, perm, static_cast<const W*>(src), static_cast<W*>(dst));
    };
    switch (words) {
        case 1: launch(permute_rows_kernel<W, 1>); break;
        case 2: launch(permute_rows_kernel<W, 2>); break;
        case 3: launch(permute_rows_kernel<W, 3>); break;
        case 6: launch(permute_rows_kernel<W, 6>); break;
        default: launch(permute_rows_kernel<W, 0>);
    }
}

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
struct SortPlan {
    BinP bp;
    int64_t ntiles;
    int bits, passes, width;
    bool few;  // kSortItemsFew elements per thread
    int64_t nblk, hist_len, scan_blocks;
    int64_t off_keys, off_vals, off_hist, off_scan, off_sums, bytes;
};

static int64_t align256(int64_t v) { return (v + 255) & ~int64_t(255); }

picasso_status make_binp(const picasso_spline* sd, const int32_t tile[3], BinP* bp,
                         int64_t* ntiles)
{
    picasso_status st = make_mesh(sd, &bp->mp);
    if (st) return st;
    if (!tile) return PICASSO_ERR_INVALID_ARGUMENT;
    bp->order = sd->order;
    int64_t nt_total = 1, tsize = 1;
    for (int d = 0; d < 3; ++d) {
        if (tile[d] < 1) return PICASSO_ERR_INVALID_ARGUMENT;
        bp->tile[d] = tile[d];
        bp->tshift[d] = -1;
        for (int sh = 0; sh < 31; ++sh)
            if ((1 << sh) == tile[d]) bp->tshift[d] = sh;
        bp->nb[d] = sd->mesh.periodic[d] ? sd->mesh.own_extent[d] : sd->mesh.extent[d];
        bp->nt[d] = (bp->nb[d] + tile[d] - 1) / tile[d];
        nt_total *= bp->nt[d];
        tsize *= tile[d];
    }
    const int64_t nkeys = nt_total * tsize;
    if (nkeys >= 0xFFFFFFFFLL) return PICASSO_ERR_OUT_OF_RANGE;
    bp->tsize = (uint32_t)tsize;
    bp->nkeys = (uint32_t)nkeys;
    *ntiles = nt_total;
    return PICASSO_OK;
}

static picasso_status make_plan(const picasso_spline* sd, int64_t n, const int32_t tile[3],
                                SortPlan* pl)
{
    if (!sd || !tile || n < 0 || n > 0xFFFFFFFELL) return PICASSO_ERR_INVALID_ARGUMENT;
    picasso_status st = make_binp(sd, tile, &pl->bp, &pl->ntiles);
    if (st) return st;
    const int64_t nkeys = pl->bp.nkeys;
    int bits = 1;
    while ((int64_t(1) << bits) <= nkeys) ++bits;  // keys are in [0, nkeys]
    pl->bits = bits;
    pl->passes = (bits + kMaxDigitBits - 1) / kMaxDigitBits;
    pl->width = (bits + pl->passes - 1) / pl->passes;
    pl->few = n < int64_t(148) * kSortThreads * kSortItems;
    const int64_t tile_len = kSortThreads * (pl->few ? kSortItemsFew : kSortItems);
    pl->nblk = n > 0 ? (n + tile_len - 1) / tile_len : 1;
    // the digit table (columns of 2048 elements or more), also used for the
    // per-tile work-item counts; a second one holds the digit totals
    pl->hist_len = (int64_t(1) << pl->width) * (n > 0 ? (n + 2047) / 2048 : 1);
    if (pl->hist_len < pl->ntiles + 1) pl->hist_len = pl->ntiles + 1;
    pl->scan_blocks = (pl->hist_len + kScanTile - 1) / kScanTile;
    int64_t o = 0;
    pl->off_keys = o;
    o = align256(o + 4 * (n > 0 ? n : 1));
    pl->off_vals = o;
    o = align256(o + 4 * (n > 0 ? n : 1));
    pl->off_hist = o;
    o = align256(o + 4 * pl->hist_len);
    pl->off_scan = o;
    o = align256(o + 4 * pl->hist_len);
    pl->off_sums = o;
    o = align256(o + 4 * pl->scan_blocks);
    pl->bytes = o;
    return PICASSO_OK;
}

// The radix passes over n > 0 particles: sorted keys and permutation in
// key / perm.  from_x: keys from the positions, else from key_src (clamped to
// nkeys).
template <int ITEMS>
static picasso_status radix_sort(const SortPlan& pl, int64_t n, bool from_x, const PField& x,
                                 const uint32_t* key_src, uint32_t* key, uint32_t* perm, char* ws,
                                 cudaStream_t s)
{
    if (n == 0) return PICASSO_OK;
    // (one ballot per bit: a kernel of 8 where the digits have no more)
    auto scatter = pl.width <= 8 ? radix_scatter_kernel<ITEMS, 8> : radix_scatter_kernel<ITEMS, 9>;
    const int smem = (int)(pl.width <= 8 ? sizeof(ScatterSmem<ITEMS, 8>) : sizeof(ScatterSmem<ITEMS, 9>));
    PB_CUDA_TRY(cudaFuncSetAttribute(scatter, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    const uint32_t kmax = pl.bp.nkeys;
    uint32_t* table = reinterpret_cast<uint32_t*>(ws + pl.off_hist);
    uint32_t* totals = reinterpret_cast<uint32_t*>(ws + pl.off_scan);
    // ping-pong so that the last pass writes the caller's arrays
    uint32_t* kbuf[2] = {reinterpret_cast<uint32_t*>(ws + pl.off_keys), key};
    uint32_t* vbuf[2] = {reinterpret_cast<uint32_t*>(ws + pl.off_vals), perm};
    int out = pl.passes & 1;  // buffer that the first pass writes
    const uint32_t* kin = from_x ? kbuf[1 - out] : key_src;
    const uint32_t* vin = nullptr;
    for (int pass = 0; pass < pl.passes; ++pass) {
        const int shift = pass * pl.width;
        const int bits = (shift + pl.width <= pl.bits) ? pl.width : pl.bits - shift;
        if (pass == 0 && from_x)
            radix_count_kernel<ITEMS, true><<<(unsigned)pl.nblk, kSortThreads, 0, s>>>(
                pl.bp, x, nullptr, kbuf[1 - out], n, shift, bits, table, pl.nblk, kmax);
        else
            radix_count_kernel<ITEMS, false><<<(unsigned)pl.nblk, kSortThreads, 0, s>>>(
                pl.bp, x, kin, nullptr, n, shift, bits, table, pl.nblk, kmax);
        radix_row_kernel<<<1u << bits, kSortThreads, 0, s>>>(table, pl.nblk, totals);
        scatter<<<(unsigned)pl.nblk, kSortThreads, smem, s>>>(
            kin, vin, kbuf[out], vbuf[out], n, shift, bits, table, totals, pl.nblk, kmax);
        kin = kbuf[out];
        vin = vbuf[out];
        out = 1 - out;
    }
    return PICASSO_OK;
}

}  // namespace pb

using namespace pb;

extern "C" picasso_status picasso_cell_sort_workspace(const picasso_spline* sd,
                                                      int64_t num_particles,
                                                      const int32_t tile[3], int64_t* bytes)
{
    if (!bytes) return PICASSO_ERR_INVALID_ARGUMENT;
    SortPlan pl;
    picasso_status st = make_plan(sd, num_particles, tile, &pl);
    if (st) return st;
    *bytes = pl.bytes;
    return PICASSO_OK;
}

// The sort proper.  key_src == nullptr: keys from the positions x_p;
// otherwise the first radix pass reads the caller's keys (clamped to nkeys)
// and takes the particle index as its value.
static picasso_status cell_sort_impl(const picasso_spline* sd, int64_t num_particles,
                                     const picasso_particle_field* x_p, const uint32_t* key_src,
                                     const int32_t tile[3], int32_t chunk, uint32_t* key,
                                     uint32_t* perm, int64_t* tile_offset, uint32_t* tile_items,
                                     void* workspace, int64_t workspace_bytes,
                                     picasso_bins* bins_out, const picasso_exec* exec)
{
    SortPlan pl;
    picasso_status st = make_plan(sd, num_particles, tile, &pl);
    if (st) return st;
    if (x_p && (st = validate_pfield(num_particles, *x_p, PICASSO_F64))) return st;
    if ((num_particles > 0 && (!key || !perm)) || !tile_offset || !tile_items || !workspace ||
        workspace_bytes < pl.bytes || chunk < 32)
        return PICASSO_ERR_INVALID_ARGUMENT;
    if (!x_p && num_particles > 0 && (!key_src || key_src == key || key_src == perm))
        return PICASSO_ERR_INVALID_ARGUMENT;
    if (reinterpret_cast<uintptr_t>(workspace) % 256) return PICASSO_ERR_INVALID_ARGUMENT;
    const int64_t n = num_particles;
    cudaStream_t s = stream_of(exec);
    char* ws = static_cast<char*>(workspace);
    const PField x = x_p ? make_pfield(*x_p) : PField{};
    if (n <= kSmallSort && pl.ntiles <= kSmallTiles) {
        PB_CUDA_TRY(cudaFuncSetAttribute(small_sort_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)sizeof(SmallSmem)));
        small_sort_kernel<<<1, kSmallThreads, sizeof(SmallSmem), s>>>(
            pl.bp, (int)n, x, x_p ? nullptr : key_src, pl.bits, key, perm, pl.ntiles, chunk, tile_offset,
            tile_items);
    } else {
        st = pl.few ? radix_sort<kSortItemsFew>(pl, n, x_p != nullptr, x, key_src, key, perm, ws, s)
                    : radix_sort<kSortItems>(pl, n, x_p != nullptr, x, key_src, key, perm, ws, s);
        if (st) return st;
        uint32_t* hist = reinterpret_cast<uint32_t*>(ws + pl.off_hist);
        uint32_t* sums = reinterpret_cast<uint32_t*>(ws + pl.off_sums);
        // per tile: offset and number of work items; then the items' prefix
        const int64_t m = pl.ntiles + 1;
        tile_offset_kernel<<<grid_for((m + 30) / 31 * 32, 128), 128, 0, s>>>(
            key, n, pl.ntiles, pl.bp.tsize, chunk, tile_offset, hist);
        if (pl.ntiles <= kSmallTiles) {
            scan_one_kernel<<<1, kScanThreads, 0, s>>>(hist, tile_items, (int)m);
        } else {
            const int64_t sb = (m + kScanTile - 1) / kScanTile;
            scan_reduce_kernel<<<(unsigned)sb, kScanThreads, 0, s>>>(hist, m, sums);
            scan_sums_kernel<<<1, kScanThreads, 0, s>>>(sums, sb);
            scan_apply_kernel<<<(unsigned)sb, kScanThreads, 0, s>>>(hist, tile_items, m, sums);
        }
    }
    if ((st = check_launch())) return st;
    if (bins_out) {
        for (int d = 0; d < 3; ++d) {
            bins_out->tile[d] = pl.bp.tile[d];
            bins_out->num_tiles[d] = pl.bp.nt[d];
            bins_out->bin_extent[d] = pl.bp.nb[d];
        }
        bins_out->order = sd->order;
        bins_out->location = sd->location;
        bins_out->chunk = chunk;
        bins_out->p2g_lanes = 0;
        bins_out->tile_offset = tile_offset;
        bins_out->tile_items = tile_items;
        bins_out->records = nullptr;
    }
    return PICASSO_OK;
}

extern "C" picasso_status picasso_cell_sort(const picasso_spline* sd, int64_t num_particles,
                                            picasso_particle_field x_p, const int32_t tile[3],
                                            int32_t chunk, uint32_t* key, uint32_t* perm,
                                            int64_t* tile_offset, uint32_t* tile_items,
                                            void* workspace, int64_t workspace_bytes,
                                            picasso_bins* bins_out, const picasso_exec* exec)
{
    return cell_sort_impl(sd, num_particles, &x_p, nullptr, tile, chunk, key, perm, tile_offset,
                          tile_items, workspace, workspace_bytes, bins_out, exec);
}

extern "C" picasso_status picasso_cell_sort_keys(const picasso_spline* sd, int64_t num_particles,
                                                 const uint32_t* key_in, const int32_t tile[3],
                                                 int32_t chunk, uint32_t* key, uint32_t* perm,
                                                 int64_t* tile_offset, uint32_t* tile_items,
                                                 void* workspace, int64_t workspace_bytes,
                                                 picasso_bins* bins_out,
                                                 const picasso_exec* exec)
{
    return cell_sort_impl(sd, num_particles, nullptr, key_in, tile, chunk, key, perm, tile_offset,
                          tile_items, workspace, workspace_bytes, bins_out, exec);
}

extern "C" picasso_status picasso_permute(int64_t num_particles, int32_t ncomp,
                                          const uint32_t* perm, picasso_particle_field src,
                                          picasso_particle_field dst, const picasso_exec* exec)
{
    if (num_particles < 0 || ncomp < 1 || (num_particles > 0 && !perm))
        return PICASSO_ERR_INVALID_ARGUMENT;
    picasso_status st;
    if ((st = validate_pfield(num_particles, src, PICASSO_F64, PICASSO_F32))) return st;
    if ((st = validate_pfield(num_particles, dst, src.dtype))) return st;
    if (num_particles > 0 && src.data == dst.data) return PICASSO_ERR_INVALID_ARGUMENT;
    if (num_particles == 0) return PICASSO_OK;
    cudaStream_t s = stream_of(exec);
    const int64_t esize = src.dtype == PICASSO_F64 ? 8 : 4;
    auto packed = [&](const picasso_particle_field& f) {
        return (f.vector_shift == 0 && f.tile_stride == ncomp && (f.comp_stride == 1 || ncomp == 1)) ||
               (ncomp == 1 && f.vector_shift >= 62);
    };
    if (packed(src) && packed(dst)) {
        const int64_t row = esize * ncomp;
        const uintptr_t al = reinterpret_cast<uintptr_t>(src.data) | reinterpret_cast<uintptr_t>(dst.data);
        const int64_t word = (row % 16 == 0 && al % 16 == 0) ? 16 : ((row % 8 == 0 && al % 8 == 0) ? 8 : 4);
        const int words = (int)(row / word);
        if (word == 16) launch_permute_rows<uint4>(num_particles, words, perm, src.data, dst.data, s);
        else if (word == 8) launch_permute_rows<uint2>(num_particles, words, perm, src.data, dst.data, s);
        else launch_permute_rows<uint32_t>(num_particles, words, perm, src.data, dst.data, s);
        return check_launch();
    }
    const unsigned blocks = grid_for(num_particles, 256);
    if (src.dtype == PICASSO_F64)
        permute_kernel<double><<<blocks, 256, 0, s>>>(num_particles, ncomp, perm, make_pfield(src),
                                                      make_pfield(dst));
    else
        permute_kernel<float><<<blocks, 256, 0, s>>>(num_particles, ncomp, perm, make_pfield(src),
                                                     make_pfield(dst));
    return check_launch();
}

// ---------------------------------------------------------------------------
// Spline records
// ---------------------------------------------------------------------------
// rec[p] = (t_x, t_y, t_z, key): the in-cell fraction of the particle's
// logical position along each dimension (FP32, rounded from the FP64
// position exactly as the transfer kernels round it) and its sort key for
// the bins' tile shape (the cell sort's key, stencil starts from the same
// FP64 arithmetic), so a transfer that reads the record builds the same
// spline and bin as one that reads the position.
namespace pb {

template <int ORDER>
__global__ void records_kernel(BinP bp, int64_t n, PField x, float4* rec)
{
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; p < n; p += stride) {
        int s[3];
        float t[3];
#pragma unroll
        for (int d = 0; d < 3; ++d)
            t[d] = logical_frac<ORDER>(x.get<double>(p, d), bp.mp.lo[d], bp.mp.rdx[d], s[d]);
        rec[p] = make_float4(t[0], t[1], t[2], __uint_as_float(key_from_starts(bp, s)));
    }
}

}  // namespace pb

extern "C" picasso_status picasso_spline_records(const picasso_spline* sd, int64_t num_particles,
                                                 picasso_particle_field x_p,
                                                 const picasso_bins* bins, void* records,
                                                 const picasso_exec* exec)
{
    if (!sd || !bins || num_particles < 0) return PICASSO_ERR_INVALID_ARGUMENT;
    if (bins->order != sd->order || bins->location != sd->location)
        return PICASSO_ERR_INVALID_ARGUMENT;
    BinP bp;
    int64_t ntiles = 0;
    picasso_status st = make_binp(sd, bins->tile, &bp, &ntiles);
    if (st) return st;
    for (int d = 0; d < 3; ++d)
        if (bins->num_tiles[d] != bp.nt[d] || bins->bin_extent[d] != bp.nb[d])
            return PICASSO_ERR_INVALID_ARGUMENT;
    if ((st = validate_pfield(num_particles, x_p, PICASSO_F64))) return st;
    if (num_particles == 0) return PICASSO_OK;
    if (!records || reinterpret_cast<uintptr_t>(records) % 16) return PICASSO_ERR_INVALID_ARGUMENT;
    cudaStream_t s = stream_of(exec);
    const PField x = make_pfield(x_p);
    float4* rec = static_cast<float4*>(records);
    const unsigned blocks = grid_for(num_particles, 256);
    if (sd->order == 1) records_kernel<1><<<blocks, 256, 0, s>>>(bp, num_particles, x, rec);
    else if (sd->order == 2) records_kernel<2><<<blocks, 256, 0, s>>>(bp, num_particles, x, rec);
    else records_kernel<3><<<blocks, 256, 0, s>>>(bp, num_particles, x, rec);
    return check_launch();
}

// ---------------------------------------------------------------------------
// Cell sort without allocation
// ---------------------------------------------------------------------------
// Callers that cannot allocate device memory when they sort -- an application
// that hands all of the GPU's memory to its own pool at start-up, a plugin
// hosted by such an application, or a time-critical loop that must never hit
// the allocator's latency or out-of-memory path -- get a sort whose scratch
// is a fixed array compiled into this library.  The array is
// kStaticSortScratchBytes large; every device on which the library's kernels
// are loaded holds it until the process exits.
namespace pb {

constexpr int64_t kStaticSortScratchBytes = 32LL << 20;  // 32 MiB
static __device__ __align__(256) unsigned char g_sort_scratch[kStaticSortScratchBytes];

// Device address of g_sort_scratch in the current context.  It is looked up
// on every call: the host-side name of a __device__ array is not a device
// address, and a cached address would go stale when the application resets
// the device or its primary context (the module is then loaded again and the
// array may move).  The lookup costs microseconds, small next to the sort's
// launches.
static picasso_status static_sort_scratch(void** out)
{
    void* p = nullptr;
    PB_CUDA_TRY(cudaGetSymbolAddress(&p, g_sort_scratch));
    *out = p;
    return PICASSO_OK;
}

}  // namespace pb

extern "C" picasso_status picasso_cell_sort_static(const picasso_spline* sd,
                                                   int64_t num_particles,
                                                   picasso_particle_field x_p,
                                                   const int32_t tile[3], int32_t chunk,
                                                   uint32_t* key, uint32_t* perm,
                                                   int64_t* tile_offset, uint32_t* tile_items,
                                                   picasso_bins* bins_out,
                                                   const picasso_exec* exec)
{
    SortPlan pl;
    picasso_status st = make_plan(sd, num_particles, tile, &pl);
    if (st) return st;
    if (pl.bytes > kStaticSortScratchBytes) return PICASSO_ERR_OUT_OF_RANGE;
    void* ws = nullptr;
    if ((st = static_sort_scratch(&ws))) return st;
    // Every scratch word the sort reads is written earlier in the same call,
    // so nothing needs clearing between calls.
    return picasso_cell_sort(sd, num_particles, x_p, tile, chunk, key, perm, tile_offset,
                             tile_items, ws, kStaticSortScratchBytes, bins_out, exec);
}
