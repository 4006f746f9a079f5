// Windowed count of 64- and 128-bit keys (k <= 63): first-occurrence filter and
// repeat table in shared memory.
//
// The count_routed kernel works on a bucket-sorted key array against the
// bucket's filter + table cells in global memory: every key costs a cell
// read and one or two atomics at L2 round-trip latency.  Here the keys of a
// bucket are grouped once more, by the slice of the bucket's table where
// their probe sequence starts (a window of WIN_Z cells), and one CTA per
// window stages the window's cells in shared memory, runs the filter test
// and the table insert of all its keys there, and writes the cells back:
// global traffic is the keys (read once, first occurrences written back in
// place) and each table cell read and written once per batch.
//
// The table layout and its probing rule are unchanged (one linear-probing
// table per bucket, the filter word of a key in the pad field of its first
// probe cell; src/BloomFilter.h:207-234 and src/ConcurrentMap.h:112-160 are
// the reference operations it replaces), so every other kernel (rehash,
// retry, export, histogram) reads the tables as before.  A probe sequence
// can run past its window into the next one; it never runs further than
// PROBE_LIMIT cells before the key counts as an overflow, so each window
// also stages the PROBE_LIMIT cells after it (the halo), and windows run in
// two phases (even, then odd windows of a bucket): no two CTAs of one phase
// stage the same cell.  A bucket table of at most WIN_Z cells is one window
// holding the whole table (probing wraps inside it).
//
//   subroute_count    keys per window, of every 16th chunk     (reads 8K/16)
//   window_caps, scan window ranges: estimate x 1.1 + 4 sigma + 64, in
//                     whole 64-key segments, then a spill area
//   subroute_scatter  keys into their window's range, staged    (reads 8K, writes 8K)
//                     in shared memory and written as runs; what
//                     a window cannot hold goes to the spill area
//   count_window x 2  filter + table in shared memory, per      (reads 8K + cells,
//                     64-key segment: first occurrences at the   writes L keys +
//                     front (seg_low), overflowed keys at the    cells)
//                     back (seg_fail), as count_routed leaves them
//   count_routed      the spill area's keys, in global memory
//   hist_window       merged histogram (on request): a window's     (reads cells,
//                     low.bin keys looked up in its staged cells     low.bin)
// Small batches, and a batch whose spill area overflows, take exact window
// counts (every chunk) instead: exact ranges, no spill.
//
// 128-bit keys (one device pass, 6 M reads at k = 63, 4096 buckets, 496 M keys;
// before: the global count, an initialisation beside the extraction, global
// histogram lookups): sub-routing 5.6 + count 5.7 ms against 12.1, extraction
// 5.4 -> 4.7, histogram 4.4 -> 2.8; count + histogram 25.0 -> 22.2.  Small inputs
// make too few windows of them: the engine takes them from 42 M keys on.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

#include "kc_kernels.cuh"

namespace kc {

constexpr int WIN_HALO = PROBE_LIMIT;              // cells staged after a window's own
constexpr uint32_t WIN_SINGLE = 63;                // zshift of a one-window bucket
template <int NW>
struct Win {
    static constexpr uint32_t ZSHIFT = NW == 1 ? 12 : 11;     // log2(Z)
    static constexpr int Z = 1 << ZSHIFT;                     // cells owned by one window
    static constexpr int CELLS = Z + WIN_HALO;                // staged per CTA
    static constexpr int CELL_BYTES = 8 * NW + 8;             // key, count, filter word: 73.7 / 61.4 KB a CTA
    // count_window: 128-bit keys take 56 registers; 6 M reads at k = 63 count
    // in 5.7 ms so, 6.1 with 2 CTAs of 512 threads, 6.9 with 3 of 512 (spills)
    static constexpr int THREADS = NW == 1 ? 512 : 384;
    static constexpr int CTAS = 3;                            // of count_window per SM
    static constexpr int HIST_CTAS = NW == 1 ? 3 : 2;         // of hist_window (whole cells: 73.7 / 81.9 KB)
    static constexpr int SCAT_ITEMS = NW == 1 ? 8 : 4;        // keys per thread of subroute_scatter
};
constexpr int WIN_THREADS = 512;                   // hist_window
constexpr int WIN_SEG = 64;                        // count_seg<1>(): output segment of 64 keys
constexpr int WIN_GROUP = 1;                       // segments a warp loads at once
constexpr int SUB_THREADS = 256;
constexpr int SUB_ITEMS = 16;
constexpr int SUB_CHUNK = SUB_THREADS * SUB_ITEMS; // keys per subroute CTA
constexpr int SUB_BINS = 2048;                     // windows a chunk counts in shared memory

// Windows of one bucket: global window ids [range_base, range_base + S), the
// window of a key = ((hash >> 17) & tab_mask) >> zshift (WIN_SINGLE: 0).
struct BucketWin {
    uint32_t range_base;
    uint32_t zshift;
};
struct WinInfo {
    uint32_t bucket;
    uint32_t sub;
};

// Window of a key, with the chunk's first bucket's entries held in registers
// (a chunk's keys lie in that bucket but for a few at its edges).
struct WinCache {
    uint32_t bucket;
    BucketWin w;
    uint64_t mask;
};
__device__ __forceinline__ bool key_empty(uint64_t k) { return k == EMPTY; }
__device__ __forceinline__ bool key_empty(const Key2& k) { return k.w0 == EMPTY && k.w1 == EMPTY; }
template <int NW>
__device__ __forceinline__ typename KeyOf<NW>::T empty_key() {
    if constexpr (NW == 1) return EMPTY;
    else return Key2{EMPTY, EMPTY};
}
// A routed key, read once.
__device__ __forceinline__ uint64_t stream_key(const uint64_t* p) { return __ldcs(p); }
__device__ __forceinline__ Key2 stream_key(const Key2* p) {
    const ulonglong2 v = __ldcs(reinterpret_cast<const ulonglong2*>(p));
    return Key2{v.x, v.y};
}
__device__ __forceinline__ uint64_t load_key(const uint64_t* p) { return *p; }
__device__ __forceinline__ Key2 load_key(const Key2* p) {
    const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(p);
    return Key2{v.x, v.y};
}
__device__ __forceinline__ void put_key(uint64_t* p, uint64_t k) { *p = k; }
__device__ __forceinline__ void put_key(Key2* p, const Key2& k) {
    *reinterpret_cast<ulonglong2*>(p) = make_ulonglong2(k.w0, k.w1);
}

template <class K>
__device__ __forceinline__ uint32_t window_of(const K& key, uint32_t bucket_shift, const WinCache& c,
                                              const BucketMeta* __restrict__ meta, const BucketWin* __restrict__ bw) {
    const uint32_t b = (uint32_t)(key_hi(key) >> bucket_shift);
    BucketWin w = c.w;
    uint64_t m = c.mask;
    if (b != c.bucket) {
        w = bw[b];
        m = __ldg(&meta[b].tab_mask);
    }
    const uint64_t cell = (hash_key(key) >> 17) & m;
    return w.range_base + (w.zshift >= WIN_SINGLE ? 0u : (uint32_t)(cell >> w.zshift));
}

// The sets of a multi-set batch: set s's keys start at start[s] and use the
// 256 buckets from 256 s on.  n = 0: one input.
struct SetSpan {
    const uint64_t* start;
    uint32_t n;
};
__device__ __forceinline__ uint32_t first_bucket(const SetSpan& sets, uint64_t i) {
    uint32_t lo = 0, hi = sets.n;  // the last set that starts at or before key i
    while (hi - lo > 1) {
        const uint32_t mid = (lo + hi) / 2;
        if (__ldg(sets.start + mid) <= i) lo = mid;
        else hi = mid;
    }
    return lo * 256;
}

// Smallest bucket of the chunk's keys (EMPTY keys skipped); 0xFFFFFFFF if none.
template <class K>
__device__ __forceinline__ uint32_t chunk_min_bucket(const K (&k)[SUB_ITEMS], uint32_t bucket_shift,
                                                     uint32_t* s_min) {
    uint32_t m = 0xFFFFFFFFu;
#pragma unroll
    for (int j = 0; j < SUB_ITEMS; ++j)
        if (!key_empty(k[j])) m = min(m, (uint32_t)(key_hi(k[j]) >> bucket_shift));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = min(m, __shfl_xor_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0) atomicMin(s_min, m);
    __syncthreads();
    return *s_min;
}

// Keys per window.  A chunk's keys lie in one or a few buckets (the input is
// bucket-routed), so they are counted in shared memory relative to the first
// window of the chunk's smallest bucket; windows out of that span (keys of
// the extraction's overflow area, or a chunk spanning many tiny buckets) go
// to global atomics.
template <int NW>
__global__ void __launch_bounds__(SUB_THREADS) subroute_count(const typename KeyOf<NW>::T* __restrict__ keys, uint64_t n,
                                                             const BucketMeta* __restrict__ meta,
                                                             const BucketWin* __restrict__ bw, uint32_t bucket_shift,
                                                             uint32_t chunk_stride, SetSpan sets,
                                                             uint32_t* __restrict__ win_count) {
    using K = typename KeyOf<NW>::T;
    __shared__ uint32_t hist[SUB_BINS];
    __shared__ uint32_t s_min;
    const uint64_t c0 = (uint64_t)blockIdx.x * chunk_stride * SUB_CHUNK;
    for (int i = threadIdx.x; i < SUB_BINS; i += SUB_THREADS) hist[i] = 0;
    if (threadIdx.x == 0) s_min = 0xFFFFFFFFu;
    K k[SUB_ITEMS];
#pragma unroll
    for (int j = 0; j < SUB_ITEMS; ++j) {
        const uint64_t i = c0 + (uint64_t)j * SUB_THREADS + threadIdx.x;
        k[j] = empty_key<NW>();
        if (i < n) k[j] = stream_key(keys + i);
    }
    bool split = false;  // a chunk that lies in several sets: every key by itself
    if (sets.n) {
        const uint32_t first = first_bucket(sets, c0);
        split = first != first_bucket(sets, min(c0 + SUB_CHUNK, n) - 1);
        if (!split) {
            meta += first;
            bw += first;
        }
    }
    __syncthreads();
    if (split) {
#pragma unroll 1
        for (int j = 0; j < SUB_ITEMS; ++j) {
            const uint64_t i = c0 + (uint64_t)j * SUB_THREADS + threadIdx.x;
            if (i >= n) continue;
            const K key = stream_key(keys + i);
            if (key_empty(key)) continue;
            const uint32_t b = first_bucket(sets, i);
            atomicAdd(&win_count[window_of(key, bucket_shift, WinCache{0xFFFFFFFFu, {}, 0}, meta + b, bw + b)], 1u);
        }
        return;  // block-uniform
    }
    const uint32_t bmin = chunk_min_bucket(k, bucket_shift, &s_min);
    if (bmin == 0xFFFFFFFFu) return;  // block-uniform: no key in this chunk
    const WinCache wc{bmin, bw[bmin], __ldg(&meta[bmin].tab_mask)};
    const uint32_t r0 = wc.w.range_base;
#pragma unroll
    for (int j = 0; j < SUB_ITEMS; ++j) {
        if (key_empty(k[j])) continue;
        const uint32_t r = window_of(k[j], bucket_shift, wc, meta, bw);
        if (r - r0 < (uint32_t)SUB_BINS) atomicAdd(&hist[r - r0], 1u);
        else atomicAdd(&win_count[r], 1u);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < SUB_BINS; i += SUB_THREADS)
        if (hist[i]) atomicAdd(&win_count[r0 + i], hist[i]);
}

// Window capacities (keys, whole 64-key output segments).  Exact: the
// window's key count.  Estimated from every chunk_stride-th chunk of keys:
// est = sampled x stride, capacity = est x 1.1 + 4 sqrt(est) + 64; the keys a
// window receives beyond it go to the spill area.
__global__ void window_caps(const uint32_t* __restrict__ cnt, uint64_t n, uint32_t chunk_stride,
                            uint32_t* __restrict__ cap) {
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        uint64_t c = cnt[i];
        if (chunk_stride > 1) {
            const double est = (double)c * (double)chunk_stride;
            c = (uint64_t)(est * 1.1 + 4.0 * sqrt(est) + 64.0);
        }
        cap[i] = (uint32_t)min((c + (WIN_SEG - 1)) & ~(uint64_t)(WIN_SEG - 1), (uint64_t)0xFFFFFFC0u);
    }
}

// First output segment of every set: that of its first window.
__global__ void set_window_segs(const BucketWin* __restrict__ bw, const uint64_t* __restrict__ start, uint32_t n_sets,
                                uint64_t* __restrict__ seg) {
    for (uint32_t s = blockIdx.x * blockDim.x + threadIdx.x; s < n_sets; s += gridDim.x * blockDim.x)
        seg[s] = start[bw[256 * s].range_base] / WIN_SEG;
}

// cursor = start; end = start + cap, for every window.
__global__ void window_bounds(const uint64_t* __restrict__ start, const uint32_t* __restrict__ cap, uint64_t n,
                              uint64_t* __restrict__ cursor, uint64_t* __restrict__ end) {
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        cursor[i] = start[i];
        end[i] = start[i] + cap[i];
    }
}

constexpr int SCAT_THREADS = 512;
constexpr int SCAT_BINS = 1024;                         // windows staged in shared memory
constexpr int SCAT_WARPS = SCAT_THREADS / 32;
template <int NW>
constexpr int scat_chunk() {  // 4096 keys of 64 bits, 2048 of 128
    return SCAT_THREADS * Win<NW>::SCAT_ITEMS;
}
// dynamic shared memory of subroute_scatter
template <int NW>
constexpr size_t scatter_smem_bytes() {
    return (size_t)scat_chunk<NW>() * 8 * NW + (size_t)SCAT_BINS * (8 + 8 + 4 + 4) + (size_t)scat_chunk<NW>() * 2;
}

struct ScatterArgs {
    const void* keys;
    uint64_t n;
    const BucketMeta* meta;
    const BucketWin* bw;
    uint32_t bucket_shift;
    unsigned long long* win_cursor;  // next free place of each window
    const uint64_t* win_end;         // end of each window's range
    unsigned long long* spill_cursor;
    uint64_t spill_end;
    uint32_t* spill_full;            // set when the spill area overflowed
    void* out;
    SetSpan sets;
};

// Keys into their window's range.  A chunk of 4096 keys is counted per
// window in shared memory, reserves one block per window it holds keys of
// (one global atomic per window and chunk; the part of a block past the
// window's capacity is reserved in the spill area instead), is staged in
// shared memory in window order, and leaves as contiguous runs.  Keys of
// windows outside the chunk's staged span are placed one by one.
//
// The input is bucket-routed, so all but a chunk in a thousand lies in one
// bucket: its window is then a mask and a shift of the hash.  (A chunk of the
// last bucket may hold EMPTY gap keys, whose top bits are that bucket's: it
// takes the general form.)  Bound by instruction issue and shared-memory
// wavefronts (the two scattered stores and the counter per key).  Half-size
// genome shape (1163 M keys, 18.6 GB): 6.84 -> 5.94 ms, 0.48 of the copy
// bandwidth, by the 32-bit window, five barriers instead of eight and one
// addition per key written.
template <int NW, bool SETS>
__global__ void __launch_bounds__(SCAT_THREADS, 3) subroute_scatter(ScatterArgs a) {
    extern __shared__ __align__(16) uint8_t sc_smem[];
    using K = typename KeyOf<NW>::T;
    constexpr int SCAT_ITEMS = Win<NW>::SCAT_ITEMS, SCAT_CHUNK = scat_chunk<NW>();
    const K* in = static_cast<const K*>(a.keys);
    K* out = static_cast<K*>(a.out);
    K* stage = reinterpret_cast<K*>(sc_smem);
    uint64_t* gdelta = reinterpret_cast<uint64_t*>(stage + SCAT_CHUNK);  // window l: staged place i goes to out[gdelta[l] + i],
    uint64_t* sdelta = gdelta + SCAT_BINS;   //   or, from limit[l] on, to the spill area at sdelta[l] + i
    uint32_t* hist = reinterpret_cast<uint32_t*>(sdelta + SCAT_BINS);  // counts, then staging offsets
    uint32_t* limit = hist + SCAT_BINS;
    uint16_t* stage_bin = reinterpret_cast<uint16_t*>(limit + SCAT_BINS);
    __shared__ uint32_t s_min, s_max;
    __shared__ __align__(16) uint32_t s_tot[SCAT_WARPS];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint64_t c0 = (uint64_t)blockIdx.x * SCAT_CHUNK;
    K k[SCAT_ITEMS];
#pragma unroll
    for (int j = 0; j < SCAT_ITEMS; ++j) {
        const uint64_t i = c0 + (uint64_t)j * SCAT_THREADS + tid;
        k[j] = empty_key<NW>();
        if (i < a.n) k[j] = stream_key(in + i);
    }
    for (int i = tid; i < SCAT_BINS; i += SCAT_THREADS) hist[i] = 0;
    if (tid == 0) {
        s_min = 0xFFFFFFFFu;
        s_max = 0;
    }
    __syncthreads();
    {
        // first and last bucket of the chunk, by the keys' first 32 bits;
        // EMPTY has all bits set
        uint32_t lo = 0xFFFFFFFFu, hi = 0;
#pragma unroll
        for (int j = 0; j < SCAT_ITEMS; ++j) {
            const uint32_t t = (uint32_t)(key_hi(k[j]) >> 32);
            lo = min(lo, t);
            hi = max(hi, t);
        }
        lo = __reduce_min_sync(0xffffffffu, lo);
        hi = __reduce_max_sync(0xffffffffu, hi);
        if (lane == 0) {
            atomicMin(&s_min, lo);
            atomicMax(&s_max, hi);
        }
    }
    __syncthreads();
    const uint32_t top_shift = a.bucket_shift - 32;
    const uint32_t bmin = s_min >> top_shift, bmax = s_max >> top_shift;
    const BucketMeta* meta = a.meta;
    const BucketWin* bw = a.bw;
    bool split = false;  // a chunk that lies in several sets: every key's own set, bins from the first one's windows on
    if constexpr (SETS) {
        const uint32_t first = first_bucket(a.sets, c0);
        split = first != first_bucket(a.sets, min(c0 + SCAT_CHUNK, a.n) - 1);
        meta += first;
        bw += first;
    }
    const BucketWin bwin = bw[split ? 0 : bmin];
    const uint64_t bmask = __ldg(&meta[bmin].tab_mask);
    const uint32_t r0 = bwin.range_base;
    const WinCache wc{split ? 0xFFFFFFFFu : bmin, bwin, bmask};
    auto general_window = [&](const K& key, int j) {
        if (!SETS || !split) return window_of(key, a.bucket_shift, wc, meta, bw);
        const uint32_t b = first_bucket(a.sets, c0 + (uint64_t)j * SCAT_THREADS + tid);
        return window_of(key, a.bucket_shift, wc, a.meta + b, a.bw + b);
    };
    // per key: staged bin (high 16 bits) and place inside it (low 16), or
    // FAR for a window outside the staged span (placed one by one later)
    constexpr uint32_t FAR = 0xFFFFFFFFu;
    uint32_t slot[SCAT_ITEMS];
    uint32_t bins = SCAT_BINS;
    const bool uniform = !split && bmin == bmax && bmin != (0xFFFFFFFFu >> top_shift);
    if (uniform) {
        // windows of at most 2^32 cells: 32-bit arithmetic
        const uint32_t wmask = bwin.zshift >= WIN_SINGLE ? 0u : (uint32_t)bmask;
        bins = min((uint32_t)SCAT_BINS, (wmask >> Win<NW>::ZSHIFT) + 1);
#pragma unroll
        for (int j = 0; j < SCAT_ITEMS; ++j) {
            const uint32_t l = ((uint32_t)(hash_key(k[j]) >> 17) & wmask) >> Win<NW>::ZSHIFT;
            slot[j] = l < (uint32_t)SCAT_BINS ? (l << 16) | atomicAdd(&hist[l], 1u) : FAR;
        }
    } else {
#pragma unroll
        for (int j = 0; j < SCAT_ITEMS; ++j) {
            slot[j] = FAR;
            if (key_empty(k[j])) continue;
            const uint32_t l = general_window(k[j], j) - r0;
            if (l < (uint32_t)SCAT_BINS) slot[j] = (l << 16) | atomicAdd(&hist[l], 1u);
        }
    }
    __syncthreads();
    // Exclusive scan of the bins (`per` consecutive ones per thread) -> staging
    // offsets; and the reservations: the window's block, and the spill block
    // for what does not fit.
    const uint32_t per = (bins + SCAT_THREADS - 1) / SCAT_THREADS;  // 1 or 2
    uint32_t h[2] = {0, 0};
    for (uint32_t q = 0; q < per; ++q) h[q] = hist[tid * per + q];
    uint32_t x = h[0] + h[1];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) s_tot[warp] = x;
    __syncthreads();
    uint32_t before = 0, staged = 0;
#pragma unroll
    for (int w = 0; w < SCAT_WARPS; ++w) {
        const uint32_t t = s_tot[w];
        before += w < warp ? t : 0u;
        staged += t;
    }
    uint32_t off = before + x - h[0] - h[1];
    for (uint32_t q = 0; q < per; ++q) {
        const uint32_t l = tid * per + q;
        hist[l] = off;
        if (h[q]) {
            const unsigned long long g = atomicAdd(&a.win_cursor[r0 + l], (unsigned long long)h[q]);
            const uint64_t end = a.win_end[r0 + l];
            const uint32_t fit = g >= end ? 0u : (uint32_t)min((uint64_t)h[q], (uint64_t)(end - g));
            gdelta[l] = g - off;
            limit[l] = off + fit;
            if (fit < h[q]) {
                const unsigned long long sp = atomicAdd(a.spill_cursor, (unsigned long long)(h[q] - fit));
                sdelta[l] = sp - (off + fit);
                if (sp + (h[q] - fit) > a.spill_end) atomicOr(a.spill_full, 1u);
            }
        }
        off += h[q];
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < SCAT_ITEMS; ++j) {
        if (slot[j] != FAR) {
            const uint32_t l = slot[j] >> 16;
            const uint32_t pos = hist[l] + (slot[j] & 0xFFFFu);
            put_key(stage + pos, k[j]);
            stage_bin[pos] = (uint16_t)l;
        } else if (!key_empty(k[j])) {  // far window: one key at a time
            const uint32_t w = general_window(k[j], j);
            const unsigned long long g = atomicAdd(&a.win_cursor[w], 1ull);
            if (g < a.win_end[w]) {
                put_key(out + g, k[j]);
            } else {
                const unsigned long long sp = atomicAdd(a.spill_cursor, 1ull);
                if (sp < a.spill_end) put_key(out + sp, k[j]);
                else atomicOr(a.spill_full, 1u);
            }
        }
    }
    __syncthreads();
    for (uint32_t i = tid; i < staged; i += SCAT_THREADS) {
        const uint32_t l = stage_bin[i];
        const K key = load_key(stage + i);
        if (i < limit[l]) {
            put_key(out + gdelta[l] + i, key);
        } else {
            const uint64_t sp = sdelta[l] + i;
            if (sp < a.spill_end) put_key(out + sp, key);
        }
    }
}

struct WindowArgs {
    void* keys;                      // window-grouped keys (subroute_scatter's output)
    const uint64_t* win_start;       // first key of each window (multiple of WIN_SEG)
    const unsigned long long* win_fill;  // place after the last key the scatter put there
    const uint32_t* win_cap;         // capacity (multiple of WIN_SEG) of each window
    const WinInfo* wins;
    const uint32_t* order;           // windows in launch order (phase 0's, then phase 1's)
    uint32_t order_base;             // this launch's first entry of `order`
    const BucketWin* bw;
    const BucketMeta* meta;
    void* table;                     // filter words in the cells' pad fields
    uint32_t* seg_low;               // per 64-key segment, as count_routed
    uint32_t* seg_fail;
    uint32_t* bucket_overflow;
    uint32_t phase;                  // 0: one-window buckets and even windows; 1: odd windows
    // the tables hold nothing yet and are not initialised: cells that no
    // window of an earlier phase has written start EMPTY in shared memory
    uint32_t fresh;
};

// Asynchronous global -> shared copies (cp.async, L1-allocating for the
// 4- and 8-byte sizes) and the wait for all of this thread's copies.
__device__ __forceinline__ void cp_async8(void* smem, const void* gmem) {
    const uint32_t s = (uint32_t)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async4(void* smem, const void* gmem) {
    const uint32_t s = (uint32_t)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }

// One CTA per window of the current phase (the launch's list of windows).
// The first batch finds its tables uninitialised (fresh) and its windows start
// EMPTY: no initialisation pass and hardly a cell read.  Half-size genome
// shape (299 M cells): count 7.67 -> 7.31 ms, and the extraction that the
// initialisation (1.6 ms) ran beside 7.58 -> 7.05.
template <int NW>
__global__ void __launch_bounds__(Win<NW>::THREADS, Win<NW>::CTAS) count_window(WindowArgs a) {
    using K = typename KeyOf<NW>::T;
    using S = typename SlotOf<NW>::T;
    constexpr int WIN_Z = Win<NW>::Z, WIN_CELLS = Win<NW>::CELLS, WIN_THREADS = Win<NW>::THREADS;
    K* const keys = static_cast<K*>(a.keys);
    extern __shared__ __align__(16) uint8_t win_smem[];
    unsigned long long* s_key = reinterpret_cast<unsigned long long*>(win_smem);
    unsigned long long* s_key1 = s_key + WIN_CELLS;  // 128-bit keys: their second words
    uint32_t* s_cnt = reinterpret_cast<uint32_t*>(win_smem + (size_t)WIN_CELLS * 8 * NW);
    uint32_t* s_pad = s_cnt + WIN_CELLS;
    __shared__ uint32_t s_full;  // a key of this window has met a full probe window
    if (threadIdx.x == 0) s_full = 0;

    const uint32_t r = a.order[a.order_base + blockIdx.x];
    const WinInfo wi = a.wins[r];
    const BucketWin bw = a.bw[wi.bucket];
    const bool single = bw.zshift >= WIN_SINGLE;
    if ((single ? 0u : (wi.sub & 1u)) != a.phase) return;  // never: the launch lists this phase's windows
    const uint64_t k0 = a.win_start[r];
    const uint32_t capk = a.win_cap[r];
    const uint32_t cnt = (uint32_t)min((unsigned long long)capk, a.win_fill[r] - k0);
    const uint32_t nseg = (cnt + WIN_SEG - 1) / WIN_SEG;
    // output segments of the window's range that hold no key (estimated
    // capacity beyond what arrived) report nothing
    for (uint32_t sg = nseg + threadIdx.x; sg < capk / WIN_SEG; sg += WIN_THREADS) {
        a.seg_low[k0 / WIN_SEG + sg] = 0;
        a.seg_fail[k0 / WIN_SEG + sg] = 0;
    }
    if (cnt == 0 && !a.fresh) return;  // block-uniform; the window's cells are left as they are
    const uint64_t M = a.meta[wi.bucket].tab_mask;
    S* tab = static_cast<S*>(a.table) + a.meta[wi.bucket].tab_off;
    const uint64_t base = single ? 0 : ((uint64_t)wi.sub << bw.zshift);
    const uint32_t W = single ? (uint32_t)(M + 1) : (uint32_t)WIN_CELLS;

    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    constexpr int ITEMS = 2 * WIN_GROUP;  // keys per lane: 2 per segment
    constexpr uint32_t GSTEP = (WIN_THREADS / 32) * WIN_GROUP;
    // a warp's keys of segment group g (EMPTY past the window's keys); the
    // loads of the next group are issued before the current one is counted,
    // the first group's before the window's cells are staged
    auto load_group = [&](uint32_t g, K (&dst)[ITEMS]) {
#pragma unroll
        for (int j = 0; j < ITEMS; ++j) {
            const uint32_t idx = (g + j / 2) * WIN_SEG + (j & 1) * 32 + lane;
            dst[j] = empty_key<NW>();
            if (g < nseg && idx < cnt) dst[j] = stream_key(keys + k0 + idx);
        }
    };
    K nxt[ITEMS];
    load_group((uint32_t)warp * WIN_GROUP, nxt);

    // stage the window (wrapping at the table's end: the last window's
    // halo) with asynchronous copies straight into the shared-memory arrays,
    // every cell's copies in flight at once.  Of fresh tables only what the
    // first phase wrote is read: an odd window's first WIN_HALO cells and its
    // halo (the even windows around it); the first phase reads nothing.
    const uint32_t lead = a.fresh ? (a.phase ? (uint32_t)WIN_HALO : 0u) : W;
    for (uint32_t i = threadIdx.x; i < W; i += WIN_THREADS) {
        if (i < lead || (a.fresh && a.phase && i >= (uint32_t)WIN_Z)) {
            const S* src = tab + ((base + i) & M);
            if constexpr (NW == 1) {
                cp_async8(&s_key[i], &src->key);
                cp_async4(&s_pad[i], &src->pad);
            } else {
                cp_async8(&s_key[i], &src->w0);
                cp_async8(&s_key1[i], &src->w1);
                cp_async4(&s_pad[i], &src->pad[0]);
            }
            cp_async4(&s_cnt[i], &src->count);
        } else {
            s_key[i] = EMPTY;
            if (NW == 2) s_key1[i] = EMPTY;
            s_cnt[i] = 0;
            s_pad[i] = 0;
        }
    }
    cp_async_wait_all();
    __syncthreads();

    const uint32_t lt = (1u << lane) - 1u;
    const uint32_t limit = (uint32_t)min((uint64_t)PROBE_LIMIT, M + 1);
    for (uint32_t g = (uint32_t)warp * WIN_GROUP; g < nseg; g += GSTEP) {
        K it[ITEMS];
        uint32_t mult[ITEMS];
#pragma unroll
        for (int j = 0; j < ITEMS; ++j) {
            const uint32_t idx = (g + j / 2) * WIN_SEG + (j & 1) * 32 + lane;
            mult[j] = idx < cnt ? 1u : 0u;
            it[j] = nxt[j];
        }
        load_group(g + GSTEP, nxt);  // other segments: never written below
        __syncwarp();  // every read of these segments precedes the in-place writes
        // hot keys arrive in runs: merge equal neighbours' keys first, so the
        // shared-memory atomics of a run are one per distinct key
#pragma unroll
        for (int j = 0; j < ITEMS; ++j) {
            bool eq_next;
            if constexpr (NW == 1) {
                const uint64_t nx = __shfl_down_sync(0xffffffffu, it[j], 1);
                eq_next = nx == it[j];
            } else {
                const uint64_t n0 = __shfl_down_sync(0xffffffffu, it[j].w0, 1);
                const uint64_t n1 = __shfl_down_sync(0xffffffffu, it[j].w1, 1);
                eq_next = n0 == it[j].w0 && n1 == it[j].w1;
            }
            if (!__any_sync(0xffffffffu, eq_next && lane < 31 && mult[j] != 0)) continue;
            const uint32_t active = __ballot_sync(0xffffffffu, mult[j] != 0);
            if (mult[j]) {
                uint32_t same;
                if constexpr (NW == 1) same = __match_any_sync(active, it[j]);
                else same = __match_any_sync(active, it[j].w0) & __match_any_sync(active, it[j].w1);
                mult[j] = ((__ffs(same) - 1) == lane) ? (uint32_t)__popc(same) : 0u;
            }
        }
        uint32_t first_bits = 0, fail_bits = 0;
#pragma unroll
        for (int j = 0; j < ITEMS; ++j) {
            if (!mult[j]) continue;
            const uint64_t h = hash_key(it[j]);
            const uint32_t local = (uint32_t)(((h >> 17) & M) - base);  // < WIN_Z (or < M + 1 for one window)
            const uint32_t bits = bloom_bits32(h);
            const uint32_t old = atomicOr(&s_pad[local], bits);
            uint32_t reps = mult[j];
            if ((old & bits) != bits) {
                first_bits |= 1u << j;
                --reps;
            }
            if (!reps) continue;
            bool done = false;
            for (uint32_t p = 0; p < limit; ++p) {
                if (p && p % PROBE_CHECK == 0 && *reinterpret_cast<volatile uint32_t*>(&s_full)) break;
                const uint32_t c = single ? (uint32_t)((local + p) & M) : local + p;
                if constexpr (NW == 1) {
                    unsigned long long cur = *reinterpret_cast<volatile unsigned long long*>(&s_key[c]);
                    if (cur == EMPTY) {
                        cur = atomicCAS(&s_key[c], EMPTY, (unsigned long long)it[j]);
                        if (cur == EMPTY) cur = it[j];
                    }
                    if (cur == it[j]) {
                        atomicAdd(&s_cnt[c], reps);
                        done = true;
                        break;
                    }
                } else {
                    // a cell is claimed word by word: the first word decides
                    // who may claim the second, the second whose cell it is;
                    // a key that loses the second goes on to the next cell
                    // (neither word of a key of k <= 63 is EMPTY)
                    unsigned long long cur = *reinterpret_cast<volatile unsigned long long*>(&s_key[c]);
                    if (cur == EMPTY) {
                        cur = atomicCAS(&s_key[c], EMPTY, (unsigned long long)it[j].w0);
                        if (cur == EMPTY) cur = it[j].w0;
                    }
                    if (cur == it[j].w0) {
                        cur = *reinterpret_cast<volatile unsigned long long*>(&s_key1[c]);
                        if (cur == EMPTY) {
                            cur = atomicCAS(&s_key1[c], EMPTY, (unsigned long long)it[j].w1);
                            if (cur == EMPTY) cur = it[j].w1;
                        }
                        if (cur == it[j].w1) {
                            atomicAdd(&s_cnt[c], reps);
                            done = true;
                            break;
                        }
                    }
                }
            }
            if (!done) {
                fail_bits |= 1u << j;
                mult[j] = reps;  // occurrences still to add after the table grows
                s_full = 1u;
                a.bucket_overflow[wi.bucket] = 1u;
            }
        }
        // per 64-key segment, as count_routed: first occurrences at the front,
        // keys that met a full probe window at the back (one copy per
        // occurrence still to add)
#pragma unroll
        for (int s = 0; s < WIN_GROUP; ++s) {
            const uint32_t seg = g + s;
            if (seg >= nseg) break;  // warp-uniform
            const uint64_t s0 = k0 + (uint64_t)seg * WIN_SEG;
            const uint64_t s_end = s0 + WIN_SEG;
            uint32_t n_low = 0, n_fail = 0;
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                const int j = 2 * s + q;
                const bool first = (first_bits >> j) & 1u;
                const uint32_t lm = __ballot_sync(0xffffffffu, first);
                if (first) put_key(keys + s0 + n_low + __popc(lm & lt), it[j]);
                n_low += __popc(lm);
            }
            if (__any_sync(0xffffffffu, ((fail_bits >> (2 * s)) & 3u) != 0)) {
#pragma unroll
                for (int q = 0; q < 2; ++q) {
                    const int j = 2 * s + q;
                    const uint32_t f = ((fail_bits >> j) & 1u) ? mult[j] : 0u;
                    uint32_t fsum = f;
#pragma unroll
                    for (int o = 1; o < 32; o <<= 1) {
                        const uint32_t y = __shfl_up_sync(0xffffffffu, fsum, o);
                        if (lane >= o) fsum += y;
                    }
                    const uint32_t wtot = __shfl_sync(0xffffffffu, fsum, 31);
                    const uint32_t my0 = n_fail + fsum - f;
                    for (uint32_t rr = 0; rr < f; ++rr) put_key(keys + s_end - 1 - (my0 + rr), it[j]);
                    n_fail += wtot;
                }
            }
            if (lane == 0) {
                a.seg_low[s0 / WIN_SEG] = n_low;
                a.seg_fail[s0 / WIN_SEG] = n_fail;
            }
        }
    }
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < W; i += WIN_THREADS) {
        ulonglong2* cell = reinterpret_cast<ulonglong2*>(tab + ((base + i) & M));
        const uint64_t cp = (uint64_t)s_cnt[i] | ((uint64_t)s_pad[i] << 32);
        if constexpr (NW == 1) {
            __stcg(cell, make_ulonglong2(s_key[i], cp));
        } else {
            __stcg(cell, make_ulonglong2(s_key[i], s_key1[i]));
            __stcg(cell + 1, make_ulonglong2(cp, 0));
        }
    }
}

template <int NW>
constexpr size_t window_smem_bytes() {
    return (size_t)Win<NW>::CELLS * Win<NW>::CELL_BYTES;
}

// ------------------------------------------------------ merged histogram
//
// The histogram pass of a one-batch windowed count whose tables have not
// grown: a window's first occurrences lie together in low.bin (the packed
// segments of its key range), so a CTA stages the window's cells and looks
// its low.bin keys up in shared memory; every cell and every low.bin record
// is read once.  A key found in the window's own cells marks its cell, whose
// count is then histogrammed with the key in low.bin added; one found in the
// halo (the next window's cells) moves its histogram entry up by one.
// Three CTAs share an SM so that one stages while others look up.  Half-size
// genome shape (321 M low.bin keys, 299 M cells, 8.0 GB): 2.5 ms, 0.49 of the
// copy bandwidth, against 22.0 ms for global lookups that marked the cells.
// Each lane probes on its own here: a vote per probe round (as lookup_low
// has) cost more than the divergence, 3.4 ms.
struct HistWindowArgs {
    const uint8_t* low;
    uint64_t n_low;
    const uint64_t* prefix;      // first low.bin record of every 64-key segment
    uint64_t nsegs, spill_seg;   // segments; the first one after the windows' ranges
    const uint64_t* win_start;
    uint64_t n_wins;
    const WinInfo* wins;
    const BucketWin* bw;
    const BucketMeta* meta;
    const void* table;
    uint32_t k, lo, hi;
    unsigned long long* gh;
    unsigned long long* extra;   // += table keys - low.bin keys found
};

__device__ __forceinline__ uint64_t cell_key(const Slot1& c) { return c.key; }
__device__ __forceinline__ Key2 cell_key(const Slot2& c) { return Key2{c.w0, c.w1}; }
__device__ __forceinline__ uint32_t& mark_of(Slot1& c) { return c.pad; }
__device__ __forceinline__ uint32_t& mark_of(Slot2& c) { return c.pad[0]; }
__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
    const uint32_t s = (uint32_t)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gmem) : "memory");
}

// dynamic shared memory of hist_window: whole cells
template <int NW>
constexpr size_t hist_window_smem() {
    return (size_t)Win<NW>::CELLS * sizeof(typename SlotOf<NW>::T);
}

template <int NW>
__global__ void __launch_bounds__(WIN_THREADS, Win<NW>::HIST_CTAS) hist_window(HistWindowArgs a) {
    using K = typename KeyOf<NW>::T;
    using S = typename SlotOf<NW>::T;
    constexpr int WIN_Z = Win<NW>::Z, WIN_CELLS = Win<NW>::CELLS;
    extern __shared__ __align__(16) uint8_t win_smem[];
    S* s_cell = reinterpret_cast<S*>(win_smem);
    __shared__ uint32_t sh[HIST_SMEM];
    __shared__ unsigned long long s_extra;
    for (int i = threadIdx.x; i < HIST_SMEM; i += WIN_THREADS) sh[i] = 0;
    if (threadIdx.x == 0) s_extra = 0;
    const uint32_t full = a.k / 32, tail_bytes = (2 * (a.k % 32) + 7) / 8, P = full * 8 + tail_bytes;
    constexpr int IT = 4 / NW;  // low.bin keys a thread holds at once
    long long extra = 0;
    uint32_t alone = 0;  // low.bin keys no table holds
    for (uint64_t r = blockIdx.x; r < a.n_wins; r += gridDim.x) {
        const WinInfo wi = a.wins[r];
        const BucketWin bw = a.bw[wi.bucket];
        const bool single = bw.zshift >= WIN_SINGLE;
        const uint64_t M = a.meta[wi.bucket].tab_mask;
        const S* tab = static_cast<const S*>(a.table) + a.meta[wi.bucket].tab_off;
        const uint64_t base = single ? 0 : ((uint64_t)wi.sub << bw.zshift);
        const uint32_t own = single ? (uint32_t)(M + 1) : (uint32_t)WIN_Z;
        const uint32_t W = single ? own : (uint32_t)WIN_CELLS;
        for (uint32_t i = threadIdx.x; i < W; i += WIN_THREADS) {
            const S* src = tab + ((base + i) & M);
            cp_async16(&s_cell[i], src);
            if constexpr (NW == 2) cp_async16(reinterpret_cast<uint4*>(&s_cell[i]) + 1, reinterpret_cast<const uint4*>(src) + 1);
        }
        const uint64_t l0 = low_at(a.prefix, a.nsegs, a.win_start[r] / WIN_SEG, a.n_low);
        const uint64_t l1 = low_at(a.prefix, a.nsegs, r + 1 < a.n_wins ? a.win_start[r + 1] / WIN_SEG : a.spill_seg,
                                   a.n_low);
        cp_async_wait_all();
        __syncthreads();
        // the pad field (the count's filter bits) becomes the cell's mark
        for (uint32_t i = threadIdx.x; i < own; i += WIN_THREADS) mark_of(s_cell[i]) = 0;
        __syncthreads();
        const uint32_t limit = (uint32_t)min((uint64_t)PROBE_LIMIT, M + 1);
        for (uint64_t i0 = l0; i0 < l1; i0 += IT * WIN_THREADS) {
            K key[IT];
#pragma unroll
            for (int j = 0; j < IT; ++j) {
                const uint64_t i = i0 + j * WIN_THREADS + threadIdx.x;
                key[j] = empty_key<NW>();
                if (i < l1) key[j] = load_low<NW>(a.low, i, P, full, tail_bytes);
            }
#pragma unroll
            for (int j = 0; j < IT; ++j) {
                if (key_empty(key[j])) continue;
                const uint64_t local64 = ((hash_key(key[j]) >> 17) & M) - base;
                if (local64 >= own) continue;  // never: the window's own low.bin records
                const uint32_t local = (uint32_t)local64;
                uint32_t c = local;
                K cur = cell_key(s_cell[c]);
                for (uint32_t p = 1; p < limit && !same_key(cur, key[j]) && !key_empty(cur); ++p) {
                    c = single ? (uint32_t)((local + p) & M) : local + p;
                    cur = cell_key(s_cell[c]);
                }
                if (!same_key(cur, key[j])) {
                    ++alone;
                    continue;
                }
                --extra;
                if (c < own) {
                    mark_of(s_cell[c]) = 1;
                } else {
                    const uint32_t n = s_cell[c].count;
                    hist_add(sh, a.gh, n, -1, a.lo, a.hi);
                    hist_add(sh, a.gh, (uint64_t)n + 1, 1, a.lo, a.hi);
                }
            }
        }
        __syncthreads();
        for (uint32_t i = threadIdx.x; i < own; i += WIN_THREADS) {
            if (key_empty(cell_key(s_cell[i]))) continue;
            ++extra;
            hist_add(sh, a.gh, (uint64_t)s_cell[i].count + mark_of(s_cell[i]), 1, a.lo, a.hi);
        }
        __syncthreads();  // the cells are overwritten by the next window's
    }
    if (a.lo <= 1 && alone) hist_add(sh, a.gh, 1, (int)alone, a.lo, a.hi);
    block_add(a.extra, extra, &s_extra);
    hist_flush(sh, a.gh, a.lo, a.hi);
}

}  // namespace kc
