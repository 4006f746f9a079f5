// Root-record radix sort (replaces sort/ExportRecordRadixSort.h:19-269), and
// the same sort over bare keys (post-processing's sorted low keys).
//
// The reference's LSD radix sort orders ExportRecord<N> by key with 8-bit
// digits, skipping bits shared by a leaf; here the records of all 256 root
// files sit in one array grouped by root id = top 8 key bits, so one stable
// LSD sort over the key's 2k significant bits orders every root file by key
// and keeps the grouping (the last pass is over the most significant bits).
//
// One pass = upsweep (per-tile digit histogram, digit-major) -> exclusive
// scan -> downsweep (stable rank inside the tile, scatter).  Stable ranking:
// a tile of 256 threads x ITEMS records is processed in ITEMS rounds of 256
// consecutive records; inside a round, __match_any_sync ranks equal digits
// within a warp and per-warp digit counts in shared memory order the warps.
//
// n records are told apart by little more than log2(n) leading key bits, so
// the passes go over the leading digits only (log2(n) + 8 bits, whole digits:
// 4 of 8 passes for 12 M keys of k = 31, 4 of 16 for k = 63), and the few runs
// of records that agree in all of those are sorted by the rest of the key
// where they lie: short runs by a thread, runs up to WARP_RUN by a warp and up
// to LONG_RUN by a block in shared memory.  Longer runs (many distinct keys
// behind one long common prefix, as poly-A tails make) are put together and
// take the passes over all digits by themselves; where they are many or hold
// half of the records, all records do.  11.7 M records of k = 31: 2.20 ms over all digits, 1.35 over four
// and the runs (high-coverage repeats with errors make ~100,000 of them).

#include <algorithm>
#include <cstdint>
#include <string>
#include <utility>
#include <vector>

#include <cuda_runtime.h>

#include "../../include/kmer_count.h"
#include "kc_internal.h"
#include "kc_scan.cuh"

namespace {

constexpr int SORT_THREADS = 256;
constexpr int SORT_ITEMS = 8;
constexpr int SORT_TILE = SORT_THREADS * SORT_ITEMS;
constexpr int RADIX = 256;

thread_local std::string g_sort_err;

// Digit `pass` of a record: bits [lowbit + 8*pass, +8) of the key taken as
// one (64*NW)-bit number (word 0 most significant).
template <int NW>
__device__ __forceinline__ uint32_t digit_of(const uint64_t* rec, uint32_t bit) {
    if constexpr (NW == 1) {
        return (uint32_t)(rec[0] >> bit) & 0xFFu;
    } else if constexpr (NW == 2) {
        // 128-bit key: w0 = rec[0] (high), w1 = rec[1] (low)
        if (bit >= 64) return (uint32_t)(rec[0] >> (bit - 64)) & 0xFFu;
        if (bit + 8 <= 64) return (uint32_t)(rec[1] >> bit) & 0xFFu;
        return (uint32_t)((rec[1] >> bit) | (rec[0] << (64 - bit))) & 0xFFu;
    } else {
        // 256-bit key: rec[0] high .. rec[3] low; a digit may straddle two words
        const uint32_t wi = 3 - (bit >> 6), sh = bit & 63;
        uint64_t v = rec[wi] >> sh;
        if (sh > 56 && wi > 0) v |= rec[wi - 1] << (64 - sh);
        return (uint32_t)v & 0xFFu;
    }
}

// A record of W 64-bit words whose first NW words are the key: an
// ExportRecord<NW> (W = NW + 1: key words, then count|pad) or a bare key
// (W = NW).
template <int W>
struct Rec {
    uint64_t w[W];
};

template <int NW, int W>
__global__ void __launch_bounds__(SORT_THREADS) upsweep(const Rec<W>* __restrict__ in, uint64_t n, uint32_t bit,
                                                         uint32_t* __restrict__ hist, uint64_t n_tiles) {
    __shared__ uint32_t h[RADIX];
    h[threadIdx.x] = 0;
    __syncthreads();
    const uint64_t t0 = (uint64_t)blockIdx.x * SORT_TILE;
#pragma unroll
    for (int r = 0; r < SORT_ITEMS; ++r) {
        const uint64_t i = t0 + (uint64_t)r * SORT_THREADS + threadIdx.x;
        if (i < n) atomicAdd(&h[digit_of<NW>(in[i].w, bit)], 1u);
    }
    __syncthreads();
    hist[(uint64_t)threadIdx.x * n_tiles + blockIdx.x] = h[threadIdx.x];
}

template <int NW, int W>
__global__ void __launch_bounds__(SORT_THREADS) downsweep(const Rec<W>* __restrict__ in, Rec<W>* __restrict__ out,
                                                           uint64_t n, uint32_t bit, const uint64_t* __restrict__ offs,
                                                           uint64_t n_tiles) {
    __shared__ uint32_t base[RADIX];                        // running count per digit inside the tile
    __shared__ uint32_t wcnt[SORT_THREADS / 32][RADIX];     // per-warp digit counts of the round
    __shared__ unsigned long long goff[RADIX];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    base[tid] = 0;
    goff[tid] = offs[(uint64_t)tid * n_tiles + blockIdx.x];
    const uint64_t t0 = (uint64_t)blockIdx.x * SORT_TILE;
    const uint32_t lt = (1u << lane) - 1u;
    for (int r = 0; r < SORT_ITEMS; ++r) {
#pragma unroll
        for (int w = 0; w < SORT_THREADS / 32; ++w) wcnt[w][tid] = 0;
        __syncthreads();
        const uint64_t i = t0 + (uint64_t)r * SORT_THREADS + tid;
        const bool valid = i < n;
        Rec<W> rec;
        uint32_t d = 0, rank_in_warp = 0;
        const uint32_t active = __ballot_sync(0xffffffffu, valid);
        if (valid) {
            rec = in[i];
            d = digit_of<NW>(rec.w, bit);
            const uint32_t same = __match_any_sync(active, d);
            rank_in_warp = __popc(same & lt);
            if (rank_in_warp == 0) wcnt[warp][d] = __popc(same);
        }
        __syncthreads();
        // thread `tid` owns digit tid: exclusive prefix over warps
        uint32_t run = 0;
#pragma unroll
        for (int w = 0; w < SORT_THREADS / 32; ++w) {
            const uint32_t c = wcnt[w][tid];
            wcnt[w][tid] = run;
            run += c;
        }
        __syncthreads();
        if (valid) out[goff[d] + base[d] + wcnt[warp][d] + rank_in_warp] = rec;
        __syncthreads();
        base[tid] += run;
    }
}

constexpr uint32_t SHORT_RUN = 16;     // records a thread sorts in place
constexpr uint32_t WARP_RUN = 128;     // records a warp sorts in shared memory
constexpr uint32_t LONG_RUN = 1024;    // records a block sorts in shared memory
constexpr uint64_t LONG_LIST = 256;    // longer runs that are sorted apart, one for every 2^16 records at most:
                                       // a run's two copies cost as much as the passes over so many
constexpr uint64_t PREFIX_MIN = 1ull << 16;  // smaller sorts are a few launches either way

template <int NW>
__device__ __forceinline__ bool key_less(const uint64_t* a, const uint64_t* b) {
#pragma unroll
    for (int w = 0; w < NW; ++w)
        if (a[w] != b[w]) return a[w] < b[w];
    return false;
}

// Runs of records that agree in the leading `bits` key bits (at most 64),
// found by their first record; runs longer than SHORT_RUN go to the list,
// which has room for them all (n / 8 entries).
struct RunList {
    unsigned long long* warp;   // runs longer than SHORT_RUN, by first record
    unsigned long long* block;  // of these, runs longer than WARP_RUN
    unsigned long long* longer;  // runs longer than LONG_RUN: first record, length (LONG_LIST pairs)
    unsigned long long* count;   // [0], [1], [2]: entries of the lists ([2] may exceed LONG_LIST)
};

template <int NW, int W>
__global__ void __launch_bounds__(SORT_THREADS) sort_runs(Rec<W>* __restrict__ r, uint64_t n, uint32_t bits, RunList list) {
    const uint32_t drop = 64 - bits;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i + 1 < n; i += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t top = r[i].w[0] >> drop;
        if (r[i + 1].w[0] >> drop != top || (i && r[i - 1].w[0] >> drop == top)) continue;
        uint32_t len = 2;
        while (len <= SHORT_RUN && i + len < n && r[i + len].w[0] >> drop == top) ++len;
        if (len > SHORT_RUN) {
            list.warp[atomicAdd(list.count, 1ull)] = i;
            continue;
        }
        for (uint32_t a = 1; a < len; ++a) {  // insertion sort
            const Rec<W> x = r[i + a];
            uint32_t b = a;
            for (; b > 0; --b) {
                const Rec<W> y = r[i + b - 1];
                if (!key_less<NW>(x.w, y.w)) break;
                r[i + b] = y;
            }
            if (b != a) r[i + b] = x;
        }
    }
}

// Bitonic sort of s[0..size) (a power of two) by the threads t, t + step, ...;
// `sync` orders the steps.
template <int NW, int W, class Sync>
__device__ __forceinline__ void bitonic(Rec<W>* s, uint32_t size, uint32_t first, uint32_t step, Sync sync) {
    for (uint32_t k = 2; k <= size; k *= 2)
        for (uint32_t j = k / 2; j > 0; j /= 2) {
            for (uint32_t t = first; t < size; t += step) {
                const uint32_t o = t ^ j;
                if (o > t && key_less<NW>(s[(t & k) ? t : o].w, s[(t & k) ? o : t].w)) {
                    const Rec<W> x = s[t];
                    s[t] = s[o];
                    s[o] = x;
                }
            }
            sync();
        }
}

// A warp per listed run: its length, then a bitonic sort; longer runs to the
// block list.
template <int NW, int W>
__global__ void __launch_bounds__(128) sort_warp_runs(Rec<W>* __restrict__ r, uint64_t n, uint32_t bits, RunList list) {
    __shared__ Rec<W> smem[4][WARP_RUN];
    const uint32_t drop = 64 - bits, lane = threadIdx.x & 31;
    Rec<W>* s = smem[threadIdx.x >> 5];
    const uint64_t runs = list.count[0];
    for (uint64_t q = (uint64_t)blockIdx.x * 4 + (threadIdx.x >> 5); q < runs; q += (uint64_t)gridDim.x * 4) {
        const uint64_t i = list.warp[q];
        const uint64_t top = r[i].w[0] >> drop;
        uint32_t len = 0;
        for (uint32_t j = 0; j <= WARP_RUN; j += 32) {
            const bool in = i + j + lane < n && r[i + j + lane].w[0] >> drop == top;
            const uint32_t m = __ballot_sync(0xffffffffu, in);
            len += m == 0xffffffffu ? 32 : __ffs(~m) - 1;
            if (m != 0xffffffffu) break;
        }
        if (len > WARP_RUN) {
            if (lane == 0) list.block[atomicAdd(list.count + 1, 1ull)] = i;
            continue;
        }
        uint32_t size = 32;
        while (size < len) size *= 2;
        for (uint32_t j = lane; j < size; j += 32) {
            if (j < len) s[j] = r[i + j];
            else
                for (int w = 0; w < W; ++w) s[j].w[w] = ~0ull;  // after every key
        }
        __syncwarp();
        bitonic<NW, W>(s, size, lane, 32, [] { __syncwarp(); });
        for (uint32_t j = lane; j < len; j += 32) r[i + j] = s[j];
        __syncwarp();
    }
}

// A block per run of the block list.
template <int NW, int W>
__global__ void __launch_bounds__(SORT_THREADS) sort_long_runs(Rec<W>* __restrict__ r, uint64_t n, uint32_t bits,
                                                               RunList list) {
    __shared__ Rec<W> s[LONG_RUN];
    __shared__ uint32_t s_len;
    const uint32_t drop = 64 - bits;
    const uint64_t runs = list.count[1];
    for (uint64_t q = blockIdx.x; q < runs; q += gridDim.x) {
        const uint64_t i = list.block[q];
        const uint64_t top = r[i].w[0] >> drop;
        if (threadIdx.x == 0) s_len = LONG_RUN + 1;
        __syncthreads();
        for (uint32_t j = threadIdx.x; j <= LONG_RUN; j += SORT_THREADS)
            if (i + j >= n || r[i + j].w[0] >> drop != top) atomicMin(&s_len, j);
        __syncthreads();
        const uint32_t len = s_len;
        __syncthreads();
        if (len > LONG_RUN) {  // block-uniform
            if (threadIdx.x == 0) {
                uint64_t lo = i + LONG_RUN, hi = n;  // the last record of the run lies in [lo, hi)
                while (hi - lo > 1) {
                    const uint64_t mid = lo + (hi - lo) / 2;
                    if (r[mid].w[0] >> drop == top) lo = mid;
                    else hi = mid;
                }
                const unsigned long long at = atomicAdd(list.count + 2, 1ull);
                if (at < LONG_LIST) {
                    list.longer[2 * at] = i;
                    list.longer[2 * at + 1] = lo + 1 - i;
                }
            }
            continue;
        }
        uint32_t size = 32;
        while (size < len) size *= 2;
        for (uint32_t j = threadIdx.x; j < size; j += SORT_THREADS) {
            if (j < len) s[j] = r[i + j];
            else
                for (int w = 0; w < W; ++w) s[j].w[w] = ~0ull;  // after every key
        }
        __syncthreads();
        bitonic<NW, W>(s, size, threadIdx.x, SORT_THREADS, [] { __syncthreads(); });
        for (uint32_t j = threadIdx.x; j < len; j += SORT_THREADS) r[i + j] = s[j];
        __syncthreads();
    }
}

template <int NW, int W>
int sort_impl(void* records, uint64_t n, uint32_t k, const KcSortScratch& w, cudaStream_t st, uint64_t* launches) {
    using R = Rec<W>;
    const uint32_t key_bits = 2 * k;
    const uint32_t lowbit = 64 * NW - key_bits;
    const uint32_t passes = (key_bits + 7) / 8;
    const uint64_t n_tiles = (n + SORT_TILE - 1) / SORT_TILE;
    R* a = static_cast<R*>(records);
    R* tmp = static_cast<R*>(w.tmp);
    uint32_t* hist = static_cast<uint32_t*>(w.hist);
    uint64_t* offs = static_cast<uint64_t*>(w.offs);
    uint64_t* sums = static_cast<uint64_t*>(w.sums);
    // `count` passes over the digits of `len` records from bit `bit` on; the
    // result is in `at` (`other`: as many records of scratch)
    auto run = [&](R* at, R* other, uint64_t len, uint32_t bit, uint32_t count) {
        const uint64_t tiles = (len + SORT_TILE - 1) / SORT_TILE, hn = (uint64_t)RADIX * tiles;
        R *src = at, *dst = other;
        for (uint32_t p = 0; p < count; ++p, bit += 8) {
            upsweep<NW, W><<<tiles, SORT_THREADS, 0, st>>>(src, len, bit, hist, tiles);
            const uint64_t nb = (hn + kc::SCAN_TILE - 1) / kc::SCAN_TILE;
            kc::scan_reduce<uint32_t><<<nb, kc::SCAN_BLOCK, 0, st>>>(hist, hn, sums);
            kc::scan_sums<<<1, kc::SCAN_BLOCK, 0, st>>>(sums, nb, 0, nullptr);
            kc::scan_apply<uint32_t, uint64_t><<<nb, kc::SCAN_BLOCK, 0, st>>>(hist, hn, sums, offs);
            downsweep<NW, W><<<tiles, SORT_THREADS, 0, st>>>(src, dst, len, bit, offs, tiles);
            std::swap(src, dst);
            *launches += 5;
        }
        cudaError_t e = cudaGetLastError();
        if (e == cudaSuccess && src != at) e = cudaMemcpyAsync(at, src, len * sizeof(R), cudaMemcpyDeviceToDevice, st);
        return e;
    };
    // the listed long runs by the passes over all digits: they lie in the order
    // of their prefixes, so sorted together each is in its place
    auto run_longer = [&](const unsigned long long* list, uint64_t count) {
        std::vector<std::pair<uint64_t, uint64_t>> runs(count);
        cudaError_t e = cudaMemcpyAsync(runs.data(), list, count * 16, cudaMemcpyDeviceToHost, st);
        if (e == cudaSuccess) e = cudaStreamSynchronize(st);
        if (e != cudaSuccess) return e;
        std::sort(runs.begin(), runs.end());
        uint64_t m = 0;
        for (const auto& q : runs) m += q.second;
        if (2 * m > n) return run(a, tmp, n, lowbit, passes);
        uint64_t at = 0;
        for (const auto& q : runs) {
            if (e == cudaSuccess)
                e = cudaMemcpyAsync(tmp + at, a + q.first, q.second * sizeof(R), cudaMemcpyDeviceToDevice, st);
            at += q.second;
        }
        if (e == cudaSuccess) e = run(tmp, tmp + m, m, lowbit, passes);
        at = 0;
        for (const auto& q : runs) {
            if (e == cudaSuccess)
                e = cudaMemcpyAsync(a + q.first, tmp + at, q.second * sizeof(R), cudaMemcpyDeviceToDevice, st);
            at += q.second;
        }
        return e;
    };
    uint32_t need = 8;
    while (need < 64 && (n >> (need - 8)) != 0) ++need;  // log2(n) + 8 bits
    const uint32_t lead = (need + 7) / 8;
    cudaError_t e;
    if (n >= PREFIX_MIN && lead <= 8 && lead < passes) {
        // the lists take the place of the offsets (256 n_tiles words: at most
        // n / 17 runs after the counters) and of the digit counts (128 n_tiles
        // words: n / 129, the longer runs from the middle on)
        unsigned long long* base = reinterpret_cast<unsigned long long*>(offs);
        unsigned long long* base2 = reinterpret_cast<unsigned long long*>(hist);
        const RunList list{base + 8, base2, base2 + 64 * n_tiles, base};
        e = run(a, tmp, n, 64 * NW - 8 * lead, lead);
        if (e == cudaSuccess) e = cudaMemsetAsync(list.count, 0, 8 * sizeof(*base), st);
        if (e == cudaSuccess) {  // (the run kernels index by the counters)
            sort_runs<NW, W><<<(uint32_t)std::min<uint64_t>((n + SORT_THREADS - 1) / SORT_THREADS, 148 * 8),
                               SORT_THREADS, 0, st>>>(a, n, 8 * lead, list);
            sort_warp_runs<NW, W><<<148 * 8, 128, 0, st>>>(a, n, 8 * lead, list);
            sort_long_runs<NW, W><<<148 * 2, SORT_THREADS, 0, st>>>(a, n, 8 * lead, list);
            *launches += 3;
            e = cudaGetLastError();
        }
        unsigned long long head[3] = {0, 0, 0};
        if (e == cudaSuccess) e = cudaMemcpyAsync(head, list.count, sizeof head, cudaMemcpyDeviceToHost, st);
        if (e == cudaSuccess) e = cudaStreamSynchronize(st);
        if (e == cudaSuccess && head[2])
            e = head[2] <= std::min(LONG_LIST, n >> 16) ? run_longer(list.longer, head[2]) : run(a, tmp, n, lowbit, passes);
    } else {
        e = run(a, tmp, n, lowbit, passes);
    }
    if (e != cudaSuccess) {
        g_sort_err = cudaGetErrorString(e);
        return KC_ERR_DEVICE;
    }
    return KC_OK;
}

}  // namespace

void kc_sort_scratch_bytes(uint64_t n, uint64_t record_bytes, uint64_t* tmp, uint64_t* hist, uint64_t* offs,
                           uint64_t* sums) {
    const uint64_t n_tiles = (n + SORT_TILE - 1) / SORT_TILE;
    const uint64_t hn = (uint64_t)RADIX * n_tiles;
    *tmp = n * record_bytes;
    *hist = hn * sizeof(uint32_t);
    *offs = hn * sizeof(uint64_t);
    *sums = ((hn + kc::SCAN_TILE - 1) / kc::SCAN_TILE + 1) * sizeof(uint64_t);
}

int kc_sort_roots(void* records, uint64_t n, uint64_t record_bytes, uint32_t k, const KcSortScratch& w,
                  cudaStream_t stream, uint64_t* launches) {
    if (n < 2) return KC_OK;
    if (record_bytes == 16 && k <= 32) return sort_impl<1, 2>(records, n, k, w, stream, launches);
    if (record_bytes == 24 && k <= 64) return sort_impl<2, 3>(records, n, k, w, stream, launches);
    if (record_bytes == 40 && k <= 128) return sort_impl<4, 5>(records, n, k, w, stream, launches);
    g_sort_err = "unsupported record layout";
    return KC_ERR_INVALID;
}

int kc_sort_keys(void* keys, uint64_t n, uint32_t nw, uint32_t k, const KcSortScratch& w, cudaStream_t stream) {
    uint64_t launches = 0;
    if (n < 2) return KC_OK;
    if (nw == 1 && k <= 32) return sort_impl<1, 1>(keys, n, k, w, stream, &launches);
    if (nw == 2 && k <= 64) return sort_impl<2, 2>(keys, n, k, w, stream, &launches);
    if (nw == 4 && k <= 128) return sort_impl<4, 4>(keys, n, k, w, stream, &launches);
    g_sort_err = "unsupported key width";
    return KC_ERR_INVALID;
}

const char* kc_sort_error() { return g_sort_err.c_str(); }
