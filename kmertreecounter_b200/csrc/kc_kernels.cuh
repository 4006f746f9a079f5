// Device kernels of the B200 exact canonical k-mer counter (sm_100a).
//
// Data flow of one batch of FASTQ bytes resident in HBM:
//
//   lines_per_tile      '\n' count of every 8 KiB tile            (reads F)
//   scan                line index at each tile start
//   extract<HIST>       canonical windows -> per-bucket totals    (reads F)
//   extract<SCATTER>    canonical windows -> bucket-contiguous    (reads F,
//                       routed key array                           writes 8N*K)
//   count_routed        first-occurrence filter + repeat tables   (reads 8N*K,
//                       on the routed array, bucket by bucket:     filter and
//                       the working set of in-flight CTAs stays    tables stay
//                       within one or two buckets, i.e. in L2      L2-resident)
//   grow_init,          after the host grew the overflowed buckets' tables
//   grow_move,          (all of them in one arena growth): move their keys,
//   count_routed        then re-insert the keys that met a full table
//     (table only)      (rehash_bucket: the same for one bucket)
//   pack_low            first occurrences -> packed low.bin bytes
//   export_count,       table slots -> ExportRecord<N> grouped by root id
//   export_write_bits   (per-chunk counts and a bitmap of passing slots, then
//                       one read of only those slots)
//
// Reference semantics are restated in the comments of each kernel with the
// file:line of ScorchShana/KmerTreeCounter they follow.
#pragma once

#include <cstdint>
#include <type_traits>
#include <cuda_runtime.h>

namespace kc {

#define KC_HD __host__ __device__ __forceinline__

// Bit reversal usable from host code (unit tests) and device code.
KC_HD uint32_t brev32(uint32_t x) {
#ifdef __CUDA_ARCH__
    return __brev(x);
#else
    x = ((x >> 1) & 0x55555555u) | ((x & 0x55555555u) << 1);
    x = ((x >> 2) & 0x33333333u) | ((x & 0x33333333u) << 2);
    x = ((x >> 4) & 0x0F0F0F0Fu) | ((x & 0x0F0F0F0Fu) << 4);
    x = ((x >> 8) & 0x00FF00FFu) | ((x & 0x00FF00FFu) << 8);
    return (x >> 16) | (x << 16);
#endif
}
KC_HD uint64_t brev64(uint64_t x) {
#ifdef __CUDA_ARCH__
    return __brevll(x);
#else
    return ((uint64_t)brev32((uint32_t)x) << 32) | brev32((uint32_t)(x >> 32));
#endif
}
KC_HD uint32_t popc32(uint32_t x) {
#ifdef __CUDA_ARCH__
    return (uint32_t)__popc(x);
#else
    return (uint32_t)__builtin_popcount(x);
#endif
}

// Position of the r-th (0-based) set bit of x, by halving with popcounts;
// always 0..31 (the export's bitmap walk).
KC_HD uint32_t nth_set_bit(uint32_t x, uint32_t r) {
    uint32_t pos = 0, c;
    c = popc32(x & 0xFFFFu);
    if (r >= c) { r -= c; pos += 16; x >>= 16; }
    c = popc32(x & 0xFFu);
    if (r >= c) { r -= c; pos += 8; x >>= 8; }
    c = popc32(x & 0xFu);
    if (r >= c) { r -= c; pos += 4; x >>= 4; }
    c = popc32(x & 0x3u);
    if (r >= c) { r -= c; pos += 2; x >>= 2; }
    if (r >= (x & 1u)) pos += 1;
    return pos;
}

constexpr int EXT_THREADS = 256;                     // extraction CTA
constexpr int EXT_BPT = 32;                          // bytes per thread
constexpr int EXT_TILE = EXT_THREADS * EXT_BPT;      // 8 KiB per CTA
constexpr int HALO = 128;                            // bytes kept before a batch (k - 1 <= 127)
constexpr int HALO_SEGS = HALO / 32;                 // extraction segments of halo
// The 256-bucket scatter staging area holds extraction to 4 CTAs per SM;
// telling the compiler so lets it use up to 64 registers (measured 6% faster
// than its default of 32).
constexpr int EXT_MIN_CTAS = 4;
// Bucket regions of a batch of at least EST_MIN_TILES tiles are sized from a
// histogram of every EST_STRIDE-th tile instead of all of them.
constexpr uint32_t EST_STRIDE = 32;
constexpr uint64_t EST_MIN_TILES = 4096;
constexpr int CNT_THREADS = 256;                     // count CTA
constexpr uint64_t EMPTY = ~0ull;                    // never a canonical key
constexpr int PROBE_LIMIT = 512;                     // linear-probe bound before overflow
// Probes between two looks at whether the bucket has overflowed already, and
// the lockstep rounds of count_routed after which a key's window is probed by
// the whole warp (insert_far).  A bucket that overflows is grown and its failed
// keys are inserted then, so once one key has met a full probe window the
// others of the bucket need not walk theirs to the end.  100,000 reads at 3x
// coverage, whose tables fill up: count stage 5.6 ms with every key walking 512
// cells, 0.70 ms in windows and 0.79 by count_routed with an early end.
constexpr uint32_t PROBE_CHECK = 32;

// One 128-bit key word pair in the reference's kmer<2> order: w0 = data[0]
// (most significant, first bases), w1 = data[1].
struct Key2 {
    uint64_t w0, w1;
};
// 256-bit key (k = 65..128), kmer<4> order: w0 most significant.
struct Key4 {
    uint64_t w0, w1, w2, w3;
};

// One extraction tile of a multi-set batch: bytes [start, min(start + 8 KiB,
// end)) of read set `set`, whose k-mers are counted with `k` into buckets
// [set * n_buckets, (set + 1) * n_buckets).  first_tile = index of the set's
// first tile (line numbers restart there; no halo before it).
struct SetTile {
    uint64_t start, end;
    uint32_t set, k, first_tile, pad;
};

// Per-bucket placement of the first-occurrence filter and the repeat table.
struct BucketMeta {
    uint64_t bloom_off;   // in 64-bit words
    uint64_t bloom_mask;  // words - 1 (power of two)
    uint64_t tab_off;     // in slots
    uint64_t tab_mask;    // slots - 1 (power of two)
};

// Repeat-table slots.  Slot1 has exactly the ExportRecord<1> layout
// {u64 key; u32 count; u32 pad} (src/definition.h:159-163).
struct __align__(16) Slot1 {
    uint64_t key;
    uint32_t count;
    uint32_t pad;
};
// 256-bit keys have no CAS of their width.  For k <= 127 the count claims a
// slot half by half (table_add4_halves).  At k = 128 a half can be all ones,
// and a slot is claimed by a CAS of `state` (SLOT_EMPTY -> SLOT_WRITING): the
// owner writes the key and the first count and publishes them with a release
// of state = SLOT_READY.  A thread that meets a SLOT_WRITING slot waits for it
// (bounded) before comparing.  Either way a used slot is SLOT_READY at the
// kernel's end, and an unused one has EMPTY words.
constexpr uint32_t SLOT_EMPTY = 0, SLOT_WRITING = 1, SLOT_READY = 2;
constexpr uint32_t PUBLISH_WAIT_LIMIT = 1u << 22;  // polls before a wait counts as a device error
struct __align__(16) Slot4 {
    uint64_t w0, w1, w2, w3;
    uint32_t count;
    uint32_t state;
    uint64_t mark;  // unused, zero: keeps the slot a multiple of 16 bytes
};
struct __align__(32) Slot2 {
    uint64_t w0, w1;
    uint32_t count;
    uint32_t pad[3];
};

// ---------------------------------------------------------------- helpers

__device__ __forceinline__ uint64_t mix64(uint64_t x) {
    // 64-bit finaliser of MurmurHash3 (Appleby, public domain).
    x ^= x >> 33;
    x *= 0xff51afd7ed558ccdull;
    x ^= x >> 33;
    x *= 0xc4ceb9fe1a85ec53ull;
    x ^= x >> 33;
    return x;
}
__device__ __forceinline__ uint64_t hash_key(uint64_t k) { return mix64(k); }
__device__ __forceinline__ uint64_t hash_key(const Key2& k) {
    return mix64(k.w0 ^ mix64(k.w1 + 0x9e3779b97f4a7c15ull));
}
__device__ __forceinline__ uint64_t hash_key(const Key4& k) {
    return mix64(k.w0 ^ mix64(k.w1 ^ mix64(k.w2 ^ mix64(k.w3 + 0x9e3779b97f4a7c15ull))));
}

// Bit 7 of each byte of the result: that byte of x is zero.  Exact per byte:
// (b & 0x7F) + 0x7F carries into bit 7 unless the low seven bits are zero,
// and never out of the byte.
KC_HD uint32_t zero_bytes(uint32_t x) {
    const uint32_t t = ((x & 0x7F7F7F7Fu) + 0x7F7F7F7Fu) | x;
    return ~t & 0x80808080u;
}

// Bit 7 of byte j (j = 0..3) -> bit j of the result: the four flag bits sit
// at 7, 15, 23, 31; times 2^21 + 2^14 + 2^7 + 1 they meet at bits 28..31
// (the other products fall below bit 22 or out of the word).
KC_HD uint32_t gather_bit7(uint32_t f) { return (f * 0x00204081u) >> 28; }

// Reverse the order of the 32 two-bit bases of a word (base p -> 31-p).
KC_HD uint64_t rev_bases(uint64_t x) {
    x = brev64(x);
    return ((x >> 1) & 0x5555555555555555ull) | ((x & 0x5555555555555555ull) << 1);
}

template <int NW>
struct KeyOf;
template <>
struct KeyOf<1> {
    using T = uint64_t;
};
template <>
struct KeyOf<2> {
    using T = Key2;
};
template <>
struct KeyOf<4> {
    using T = Key4;
};

__device__ __forceinline__ uint64_t key_hi(uint64_t k) { return k; }
__device__ __forceinline__ uint64_t key_hi(const Key2& k) { return k.w0; }
__device__ __forceinline__ uint64_t key_hi(const Key4& k) { return k.w0; }

// Canonical key of the window W (the last k bases, oldest base in the high
// bits of the 2k-bit value, newest in bits 1..0).
//
// The reference keeps two registers (src/GetKmer.h:58-82):
//   F = the window bases in REVERSE read order, not complemented, left-aligned
//   C = the complemented bases in read order, left-aligned
// and emits min(F, C) compared word by word (src/GetKmer.h:181-207).  With W
// as defined here F = rev_bases(W) (left-aligned by the reversal itself) and
// C = (~W masked to 2k bits) << (64N - 2k).
KC_HD uint64_t canonical1(uint64_t W, uint32_t k) {
    const uint64_t F = rev_bases(W);
    const uint64_t C = (k == 32) ? ~W : ((~W) << (64 - 2 * k));
    return F < C ? F : C;
}
KC_HD Key2 canonical2(uint64_t Whi, uint64_t Wlo, uint32_t k) {
    // F = base-reverse of the 128-bit (Whi:Wlo); the window occupies the low
    // 2k bits so the reversal lands it left-aligned.
    Key2 F{rev_bases(Wlo), rev_bases(Whi)};
    // C = ~W in 2k bits, shifted left by 128 - 2k (k in 33..64 -> 0..62).
    const uint32_t s = 128 - 2 * k;
    const uint64_t nhi = ~Whi, nlo = ~Wlo;
    Key2 C;
    if (s == 0) {
        C.w0 = nhi;
        C.w1 = nlo;
    } else {
        C.w0 = (nhi << s) | (nlo >> (64 - s));
        C.w1 = nlo << s;
    }
    const bool f_less = (F.w0 < C.w0) || (F.w0 == C.w0 && F.w1 < C.w1);
    return f_less ? F : C;
}

// k = 65..128: the window is the 256-bit W3:W2:W1:W0 (W0 = the newest 32
// bases, oldest base highest), of which the low 2k bits are the k bases.
// F = base-reverse of all 256 bits (left-aligned by the reversal itself);
// C = (~W masked to 2k bits) << (256 - 2k); key = the lexicographic min.
KC_HD Key4 canonical4(uint64_t W0, uint64_t W1, uint64_t W2, uint64_t W3, uint32_t k) {
    const uint32_t kb = 2 * k;  // 130..256
    if (kb <= 192) {
        W3 = 0;
        if (kb < 192) W2 &= (1ull << (kb - 128)) - 1ull;
    } else if (kb < 256) {
        W3 &= (1ull << (kb - 192)) - 1ull;
    }
    const Key4 F{rev_bases(W0), rev_bases(W1), rev_bases(W2), rev_bases(W3)};
    // ~W restricted to the 2k bits
    uint64_t n0 = ~W0, n1 = ~W1, n2 = ~W2, n3 = ~W3;
    if (kb <= 192) {
        n3 = 0;
        if (kb < 192) n2 &= (1ull << (kb - 128)) - 1ull;
    } else if (kb < 256) {
        n3 &= (1ull << (kb - 192)) - 1ull;
    }
    // shift left by sh = 256 - 2k (0..126): whole words first, then bits
    const uint32_t sh = 256 - kb;
    if (sh >= 64) {
        n3 = n2;
        n2 = n1;
        n1 = n0;
        n0 = 0;
    }
    const uint32_t r = sh & 63;
    if (r) {
        n3 = (n3 << r) | (n2 >> (64 - r));
        n2 = (n2 << r) | (n1 >> (64 - r));
        n1 = (n1 << r) | (n0 >> (64 - r));
        n0 = n0 << r;
    }
    const Key4 C{n3, n2, n1, n0};
    bool f_less;
    if (F.w0 != C.w0) f_less = F.w0 < C.w0;
    else if (F.w1 != C.w1) f_less = F.w1 < C.w1;
    else if (F.w2 != C.w2) f_less = F.w2 < C.w2;
    else f_less = F.w3 < C.w3;
    return f_less ? F : C;
}

// ------------------------------------------------------------ block scans

// Exclusive scan of one uint32 per thread over a CTA of BLOCK threads.
template <int BLOCK>
__device__ __forceinline__ uint32_t block_exclusive_scan(uint32_t v, uint32_t* smem_warp, uint32_t* total) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) smem_warp[warp] = x;
    __syncthreads();
    if (warp == 0) {
        uint32_t w = lane < BLOCK / 32 ? smem_warp[lane] : 0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, w, o);
            if (lane >= o) w += y;
        }
        if (lane < BLOCK / 32) smem_warp[lane] = w;
    }
    __syncthreads();
    const uint32_t warp_prefix = warp ? smem_warp[warp - 1] : 0;
    if (total) *total = smem_warp[BLOCK / 32 - 1];
    const uint32_t r = warp_prefix + x - v;
    __syncthreads();
    return r;
}

// ------------------------------------------------ control-path transfers
//
// Counts, cursors and flags move between host and device as kernels that
// read or write mapped pinned memory, and small fills run as kernels: the
// copy engines are kept for the bulk FASTQ and output copies, behind which a
// few-byte copy would otherwise wait.

// Up to CTL_OPS of them, with nothing in between, are one launch (a launch
// per few bytes was a third of the launches of a small count): op
// blockIdx.y copies n words from src, or fills with `word` without one.
constexpr int CTL_OPS = 8;
struct CtlOp {
    uint32_t* dst;
    const uint32_t* src;
    uint64_t n;
    uint32_t word;
};
struct CtlOps {
    CtlOp op[CTL_OPS];
};
static __global__ void control_ops(const __grid_constant__ CtlOps o) {
    const CtlOp p = o.op[blockIdx.y];
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < p.n; i += (uint64_t)gridDim.x * blockDim.x)
        p.dst[i] = p.src ? p.src[i] : p.word;
}

static __global__ void fill_words(uint32_t* __restrict__ dst, uint64_t n, uint32_t v) {
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x)
        dst[i] = v;
}

// Zero n 16-byte units (16-byte aligned).
static __global__ void zero16(uint4* __restrict__ dst, uint64_t n) {
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x)
        dst[i] = make_uint4(0u, 0u, 0u, 0u);
}

// ------------------------------------------------------- FASTQ line split

// '\n' count per 8 KiB tile of the batch buf[0..n) (16-byte vector reads,
// byte reads for the ragged end).
static __global__ void lines_per_tile(const uint8_t* __restrict__ buf, uint64_t n, uint32_t* __restrict__ tile_nl) {
    __shared__ uint32_t warp_sums[EXT_THREADS / 32];
    const uint64_t tile = blockIdx.x;
    const uint64_t pos = tile * EXT_TILE + (uint64_t)threadIdx.x * EXT_BPT;
    uint32_t cnt = 0;
    if (pos < n) {
        const uint64_t rem = n - pos;
        if (rem >= 32) {
            const uint4* p = reinterpret_cast<const uint4*>(buf + pos);
            const uint4 a = __ldcs(p), b = __ldcs(p + 1);
            const uint32_t w[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
#pragma unroll
            for (int i = 0; i < 8; ++i) cnt += __popc(zero_bytes(w[i] ^ 0x0A0A0A0Au));
        } else {
            for (uint32_t j = 0; j < (uint32_t)rem; ++j) cnt += buf[pos + j] == '\n';
        }
    }
    uint32_t total;
    block_exclusive_scan<EXT_THREADS>(cnt, warp_sums, &total);
    if (threadIdx.x == 0) tile_nl[tile] = total;
}

// '\n' count of each set tile (multi-set batches).
static __global__ void lines_per_set_tile(const uint8_t* __restrict__ buf, const SetTile* __restrict__ tiles,
                                          uint32_t* __restrict__ tile_nl) {
    __shared__ uint32_t warp_sums[EXT_THREADS / 32];
    const SetTile t = tiles[blockIdx.x];
    const uint64_t pos = t.start + (uint64_t)threadIdx.x * EXT_BPT;
    uint32_t cnt = 0;
    if (pos < t.end) {
        const uint64_t rem = t.end - pos;
        if (rem >= 32) {
            const uint4* p = reinterpret_cast<const uint4*>(buf + pos);
            const uint4 a = __ldcs(p), b = __ldcs(p + 1);
            const uint32_t w[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
#pragma unroll
            for (int i = 0; i < 8; ++i) cnt += __popc(zero_bytes(w[i] ^ 0x0A0A0A0Au));
        } else {
            for (uint32_t j = 0; j < (uint32_t)rem; ++j) cnt += buf[pos + j] == '\n';
        }
    }
    uint32_t total;
    block_exclusive_scan<EXT_THREADS>(cnt, warp_sums, &total);
    if (threadIdx.x == 0) tile_nl[blockIdx.x] = total;
}

// Line index at each tile start, counted from its own set's first byte.
static __global__ void rebase_set_lines(const uint64_t* __restrict__ global_prefix, const SetTile* __restrict__ tiles,
                                        uint64_t n_tiles, uint64_t* __restrict__ tile_line) {
    for (uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; t < n_tiles; t += (uint64_t)gridDim.x * blockDim.x)
        tile_line[t] = global_prefix[t] - global_prefix[tiles[t].first_tile];
}

// ------------------------------------------------------- k-mer extraction

enum ExtractMode { HIST = 0, SCATTER = 1 };

// Classification of one thread's 32 bytes.
struct Seg {
    uint64_t codes;  // 2-bit codes, byte 0 in bits 63..62 (appending order)
    uint32_t bases;  // bit j set: byte j is A/C/G/T/U (either case)
    uint32_t nls;    // bit j set: byte j is '\n'
};

// Byte selection of the PRMT instruction: byte i of the result is byte
// (sel >> 4i) & 7 of the eight bytes y:x.
KC_HD uint32_t byte_perm(uint32_t x, uint32_t y, uint32_t sel) {
#ifdef __CUDA_ARCH__
    return __byte_perm(x, y, sel);
#else
    const uint64_t v = ((uint64_t)y << 32) | x;
    uint32_t r = 0;
    for (int i = 0; i < 4; ++i) r |= (uint32_t)((v >> (8 * ((sel >> (4 * i)) & 7))) & 0xFF) << (8 * i);
    return r;
#endif
}

// Four bytes at a time.  The 2-bit code of a base is ((c >> 1) ^ (c >> 2)) & 3
// (A=0 C=1 G=2 T/U=3, either case); any byte has such a code, and it is a base
// when it equals the letter of its code: the letter is looked up by byte
// permutation, case (0x20) is ignored, and for code 3 bit 0 too (T = 0x54,
// U = 0x55).  Newlines by the exact zero-byte test.
KC_HD Seg classify(const uint32_t (&w)[8], uint64_t valid_bytes) {
    Seg s{0, 0, 0};
    uint32_t prod[8];  // the word's four codes in byte 3
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const uint32_t x = w[i];
        const uint32_t code4 = ((x >> 1) ^ (x >> 2)) & 0x03030303u;
        // codes of bytes 4i..4i+3 -> 8 bits, byte 4i in the high pair: the
        // 2-bit fields at 0, 8, 16, 24 times 2^30 + 2^20 + 2^10 + 1 land at
        // 30, 28, 26, 24 (the other products fall below bit 22 or out)
        prod[i] = code4 * 0x40100401u;
        // the codes as selector nibbles 0..3
        const uint32_t sel = byte_perm(code4 | (code4 >> 4), 0u, 0x20u) & 0xFFFFu;
        const uint32_t letter = byte_perm(0x54474341u, 0u, sel);  // A C G T
        const uint32_t care = byte_perm(0xDEDFDFDFu, 0u, sel);
        const uint32_t isb = zero_bytes((x ^ letter) & care);
        const uint32_t isn = zero_bytes(x ^ 0x0A0A0A0Au);
        s.bases |= gather_bit7(isb) << (4 * i);
        s.nls |= gather_bit7(isn) << (4 * i);
    }
    const uint32_t chi = byte_perm(byte_perm(prod[2], prod[3], 0x37u), byte_perm(prod[0], prod[1], 0x37u), 0x5410u);
    const uint32_t clo = byte_perm(byte_perm(prod[6], prod[7], 0x37u), byte_perm(prod[4], prod[5], 0x37u), 0x5410u);
    s.codes = ((uint64_t)chi << 32) | clo;
    if (valid_bytes < 32) {
        const uint32_t keep = valid_bytes ? (0xFFFFFFFFu >> (32 - (uint32_t)valid_bytes)) : 0u;
        s.bases &= keep;
        s.nls &= keep;
    }
    return s;
}

// 32 bytes starting at p, of which only the first `avail` may be read (the
// rest read as 0).  Full segments use two 16-byte vector loads.
__device__ __forceinline__ void load32(const uint8_t* p, uint64_t avail, uint32_t (&w)[8]) {
    if (avail >= 32) {
        const uint4* q = reinterpret_cast<const uint4*>(p);
        const uint4 a = __ldcs(q), b = __ldcs(q + 1);
        w[0] = a.x; w[1] = a.y; w[2] = a.z; w[3] = a.w;
        w[4] = b.x; w[5] = b.y; w[6] = b.z; w[7] = b.w;
    } else {
#pragma unroll
        for (int i = 0; i < 8; ++i) w[i] = 0;
        for (uint32_t j = 0; j < (uint32_t)avail; ++j) w[j >> 2] |= (uint32_t)p[j] << (8 * (j & 3));
    }
}

typedef unsigned __int128 u128;

// Bit i of the result: bits [i-k+1, i] of X are all set (bits below 0 read
// as clear).  Shift-AND doubling: R_2m = R_m & (R_m << m), then one
// overlapping step to reach k exactly.
__device__ __forceinline__ u128 runs_at_least(u128 X, uint32_t k) {
    u128 R = X;
    uint32_t have = 1;
    while (2 * have <= k) {
        R &= R << have;
        have *= 2;
    }
    if (have < k) R &= R << (k - have);
    return R;
}

// The same over five segments' base bits (b0 oldest .. b4 current, 160 bits)
// for k = 65..128: bit j of the result = the k bytes ending at byte j of b4
// are all bases.
KC_HD uint32_t runs_at_least5(uint32_t b0, uint32_t b1, uint32_t b2, uint32_t b3, uint32_t b4, uint32_t k) {
    uint64_t x0 = (uint64_t)b0 | ((uint64_t)b1 << 32), x1 = (uint64_t)b2 | ((uint64_t)b3 << 32), x2 = b4;
    auto and_shifted = [&](uint32_t n) {  // X &= X << n, 1 <= n <= 64
        uint64_t y0, y1, y2;
        if (n == 64) {
            y2 = x1;
            y1 = x0;
            y0 = 0;
        } else {
            y2 = (x2 << n) | (x1 >> (64 - n));
            y1 = (x1 << n) | (x0 >> (64 - n));
            y0 = x0 << n;
        }
        x0 &= y0;
        x1 &= y1;
        x2 &= y2;
    };
    uint32_t have = 1;
    while (2 * have <= k) {
        and_shifted(have);
        have *= 2;
    }
    if (have < k) and_shifted(k - have);
    return (uint32_t)x2;
}

// runs_at_least for k <= 32: the k bytes ending at byte j of the segment with
// base bits `cur` lie in it and the segment before it (`prev`).
KC_HD uint32_t runs_at_least2(uint32_t prev, uint32_t cur, uint32_t k) {
    uint64_t R = ((uint64_t)cur << 32) | prev;
    uint32_t have = 1;
    while (2 * have <= k) {
        R &= R << have;
        have *= 2;
    }
    if (have < k) R &= R << (k - have);
    return (uint32_t)(R >> 32);
}

// Bit j: parity of the bits 0..j of x.
KC_HD uint32_t prefix_parity(uint32_t x) {
    x ^= x << 1;
    x ^= x << 2;
    x ^= x << 4;
    x ^= x << 8;
    return x ^ (x << 16);
}

// Bits of the 32 bytes that lie on sequence lines (line index = 1 mod 4),
// line0 = line index of byte 0, nls = newline bits.  The number of newlines
// before a byte, mod 4, bit by bit: its low bit is their parity, its high bit
// the parity of those that found the low bit set.
KC_HD uint32_t sequence_mask(uint32_t line0, uint32_t nls) {
    const uint32_t low = prefix_parity(nls) << 1;
    const uint32_t high = prefix_parity(nls & low) << 1;
    const uint32_t want = 1u - line0;  // mod 4
    const uint32_t w0 = (want & 1u) ? ~0u : 0u, w1 = (want & 2u) ? ~0u : 0u;
    return ~(low ^ w0) & ~(high ^ w1);
}

// Reverse the order of the nb two-bit bases in the low 2*nb bits of x.
KC_HD uint32_t rev_small(uint32_t x, uint32_t nb) {
    uint32_t r = brev32(x);
    r = ((r >> 1) & 0x55555555u) | ((r & 0x55555555u) << 1);
    return r >> (32 - 2 * nb);
}

// Window of the last k bases ending at byte j of segment s2 (segments s0,
// s1 precede it): low 64 bits and, for k > 32, the next 64 bits.
KC_HD void window_at(uint64_t s0, uint64_t s1, uint64_t s2, uint32_t j, uint64_t& lo,
                                          uint64_t& hi) {
    const uint32_t sh = 2 * (31 - j);  // 0..62
    if (sh == 0) {
        lo = s2;
        hi = s1;
    } else {
        lo = (s2 >> sh) | (s1 << (64 - sh));
        hi = (s1 >> sh) | (s0 << (64 - sh));
    }
}

// The 256-bit window of the last 128 bases ending at byte j of segment s4
// (segments s0..s3 precede it): W0 = the newest 32 bases.
KC_HD void window_at4(uint64_t s0, uint64_t s1, uint64_t s2, uint64_t s3, uint64_t s4, uint32_t j, uint64_t& W0,
                      uint64_t& W1, uint64_t& W2, uint64_t& W3) {
    const uint32_t sh = 2 * (31 - j);
    if (sh == 0) {
        W0 = s4;
        W1 = s3;
        W2 = s2;
        W3 = s1;
    } else {
        W0 = (s4 >> sh) | (s3 << (64 - sh));
        W1 = (s3 >> sh) | (s2 << (64 - sh));
        W2 = (s2 >> sh) | (s1 << (64 - sh));
        W3 = (s1 >> sh) | (s0 << (64 - sh));
    }
}

struct ExtractArgs {
    const SetTile* tiles;    // multi-set batch: per-tile descriptor (nullptr: one input)
    const uint8_t* buf;      // batch start (16-byte aligned)
    uint64_t n;              // batch bytes
    int has_halo;            // buf[-HALO..-1] are the bytes before the batch
    const uint64_t* tile_line;  // line index at each tile start
    uint32_t k;
    uint32_t bucket_shift;   // 64 - log2(n_buckets)
    uint32_t n_buckets;
    unsigned long long* bucket_count;  // HIST: per-bucket totals (accumulated)
    unsigned long long* bucket_cursor; // SCATTER: next free index per bucket
    void* routed;            // SCATTER: routed key array
    uint32_t* error;         // bit 0: a key's bucket disagreed with its reservation;
                             // bit 1: the overflow area was full (keys dropped)
    uint32_t tile_stride;    // HIST over every tile_stride-th tile only (0 or 1: all)
    // SCATTER into estimated regions: bucket b owns routed[cursor0[b], region_end[b]).
    // A CTA's run of bucket b that does not fit whole goes whole to the overflow
    // area routed[overflow_start, overflow_end) (cursor *overflow_cursor), and
    // region_fill[b] (atomicMin) records where the region stopped filling.
    // region_end == nullptr: the regions are exact (no overflow).
    const unsigned long long* region_end;
    unsigned long long* region_fill;
    unsigned long long* overflow_cursor;
    uint64_t overflow_start, overflow_end;
    // multi-set batch with estimated regions: per set s an overflow area
    // [set_ovf_start[s], set_ovf_end[s]) with cursor set_ovf_cursor[s]; the
    // region arrays are indexed by set x n_buckets + bucket
    const uint64_t* set_ovf_start;
    const uint64_t* set_ovf_end;
    unsigned long long* set_ovf_cursor;
    // HIST over the listed tiles only (nullptr: every tile_stride-th)
    const uint32_t* tile_list;
};

// Bucket of the canonical key of window (hi:lo) without building the key:
// the top B bits of min(F, C) equal min(top B bits of F, top B bits of C).
// top(F) = the newest B/2 bases reversed; top(C) = the oldest B/2 bases
// complemented.
KC_HD uint32_t bucket_of_window(uint64_t lo, uint64_t hi, uint32_t k, uint32_t B) {
    const uint32_t nb = B / 2;
    const uint32_t mask = (1u << B) - 1u;
    const uint32_t topF = k >= nb ? rev_small((uint32_t)lo & mask, nb) : (rev_small((uint32_t)lo & ((1u << (2 * k)) - 1u), k) << (B - 2 * k));
    uint32_t topC;
    const uint32_t lo_bit = 2 * k >= B ? 2 * k - B : 0;  // lowest bit of the oldest B/2 bases
    if (2 * k < B) {
        topC = ((~(uint32_t)lo) & ((1u << (2 * k)) - 1u)) << (B - 2 * k);
    } else if (lo_bit + B <= 64) {
        topC = (uint32_t)(~lo >> lo_bit) & mask;
    } else if (lo_bit >= 64) {
        topC = (uint32_t)(~hi >> (lo_bit - 64)) & mask;
    } else {
        topC = (uint32_t)(((~lo) >> lo_bit) | ((~hi) << (64 - lo_bit))) & mask;
    }
    return topF < topC ? topF : topC;
}

// ---- canonical keys from two base streams
//
// Both orientations of a window are contiguous in a stream of 2-bit codes:
// C (complemented, read order) in the stream of complemented codes, first base
// first; F (not complemented, newest base first) in the stream of codes in
// reverse order.  A tile keeps both as 32-bit words (16 bases, first one in
// the high bits), so a left-aligned key word is one funnel shift of two
// adjacent words, with no bit reversal or left alignment per key.
constexpr int TILE_SEGS = EXT_TILE / 32 + HALO_SEGS;  // segments of a tile with its halo
constexpr int C_WORDS = 2 * TILE_SEGS + 8;            // a window may read 7 words past its last base's
constexpr int STREAM_WORDS = C_WORDS + 2 * TILE_SEGS; // C stream, then F stream

KC_HD uint32_t funnel_l(uint32_t hi, uint32_t lo, uint32_t sh) {  // high word of (hi:lo) << sh, sh < 32
#ifdef __CUDA_ARCH__
    return __funnelshift_l(lo, hi, sh);
#else
    return sh ? (hi << sh) | (lo >> (32 - sh)) : hi;
#endif
}

// The codes of segment t (0 = the first halo segment) into both streams.
KC_HD void stream_put(uint32_t* sw, int t, uint64_t codes) {
    sw[2 * t] = ~(uint32_t)(codes >> 32);
    sw[2 * t + 1] = ~(uint32_t)codes;
    const uint64_t r = rev_bases(codes);
    uint32_t* f = sw + C_WORDS + 2 * (TILE_SEGS - 1 - t);
    f[0] = (uint32_t)(r >> 32);
    f[1] = (uint32_t)r;
}

// Where a k-base window that ends at byte e of the tile (halo not counted)
// starts in the streams.
struct StreamPos {
    uint32_t c, cs, f, fs;  // first word and bit shift of C, of F
};
KC_HD StreamPos stream_pos(uint32_t e, uint32_t k) {
    const uint32_t b0 = e + HALO + 1 - k;         // its first base in the C stream (k <= HALO)
    const uint32_t q = (uint32_t)EXT_TILE - 1 - e;  // its newest base in the F stream
    return StreamPos{b0 >> 4, 2 * (b0 & 15), (uint32_t)C_WORDS + (q >> 4), 2 * (q & 15)};
}

// Bits of 32-bit key word w that belong to a k-base key.
KC_HD uint32_t key_mask(uint32_t w, uint32_t k) {
    const int n = (int)(2 * k) - 32 * (int)w;
    return n >= 32 ? ~0u : (n <= 0 ? 0u : ~0u << (32 - n));
}

// The first 32 bits of the canonical key (what its bucket is taken from):
// the smaller of the orientations' first words, whichever orientation the
// rest decides for.
KC_HD uint32_t top_of_window(const uint32_t* sw, const StreamPos& p, uint32_t mask0) {
    const uint32_t f = funnel_l(sw[p.f], sw[p.f + 1], p.fs) & mask0;
    const uint32_t c = funnel_l(sw[p.c], sw[p.c + 1], p.cs) & mask0;
    return f < c ? f : c;
}

// The canonical key: the orientation with the smaller word at the first
// difference (bits past the key can differ only when all of its bits agree,
// and then either will do).
template <int NW>
KC_HD void key_of_window(const uint32_t* sw, const StreamPos& p, uint32_t k, uint64_t (&key)[NW]) {
    const uint32_t n = (2 * k + 31) / 32;  // 32-bit words that hold key bits
    bool f_less = true;
    for (uint32_t w = 0; w < n; ++w) {
        const uint32_t f = funnel_l(sw[p.f + w], sw[p.f + w + 1], p.fs);
        const uint32_t c = funnel_l(sw[p.c + w], sw[p.c + w + 1], p.cs);
        f_less = f < c;
        if (f != c) break;
    }
    const uint32_t* s = sw + (f_less ? p.f : p.c);
    const uint32_t sh = f_less ? p.fs : p.cs;
    uint32_t prev = s[0];
#pragma unroll
    for (int w = 0; w < 2 * NW; ++w) {
        uint32_t v = 0;
        if ((uint32_t)w < n) {
            const uint32_t next = s[w + 1];
            v = funnel_l(prev, next, sh) & key_mask(w, k);
            prev = next;
        }
        if (w & 1) key[w / 2] |= v;
        else key[w / 2] = (uint64_t)v << 32;
    }
}

// Canonical k-mer extraction over one 8 KiB tile per CTA.
//
// Emission rule (reference: src/FastqReader.h:140-308 + src/FastqParser.h:
// 182-455 + src/GetKmer.h:58-131): a window ending at byte p is a k-mer iff
// p lies on a sequence line (line index = 1 mod 4 counted from the start of
// the file) and the k bytes ending at p are all bases.  A window never
// crosses '\n' because '\n' is not a base, so only p's line matters.
//
// Phase A, per thread (32 bytes): classify, then a bit-parallel emit mask:
//   run of >= k bases ending at byte j (shift-AND doubling over the bases
//   of this and the preceding segments) AND byte j on a sequence line; the
//   segments that emit are listed, and their codes go to the two streams.
// Phase C, per listed segment: one warp, lane j the window ending at byte j.
//
// HIST: per-bucket totals (bucket = top bits of the canonical key, from the
// streams' first words).  SCATTER (256 buckets): every key takes its rank
// from its bucket's shared-memory counter, one reservation per bucket per CTA
// places the tile's runs in the routed array, and the keys are written in
// bucket order, as contiguous runs.
//   64-bit keys are staged in arrival order and indexed in bucket order.
//   128- and 256-bit keys, and tiles with more 64-bit keys than the staging
//   area holds, only index their positions: the first pass needs the bucket
//   alone, and the key is built from the streams when it is written, once.
//   (Staging 128-bit keys in 48 KB held 2048 of the 2300 keys of a tile of
//   150 bp reads at k = 63; the tiles that did not fit built every key twice.)
//
// The kernel is bound by shared memory (l1tex 83%, the integer pipe 65%), not by
// its bytes.  Before, bound by the integer pipe, each key came from 64-bit shifts and bit reversals of its
// segment's codes, and tiles walked all their segments: 10 M reads of 150 bp
// at k = 31 9.5 -> 7.6 ms, 6 M at k = 63 10.4 -> 5.4, 1 M of 250 bp at
// k = 101 5.2 -> 2.2.

// 64-bit keys of one tile staged in shared memory: an 8 KiB tile of 150 bp
// FASTQ holds ~3150 at k = 31, and 4 CTAs fit one SM's shared memory.
constexpr int STAGE_KEYS = 3824;
constexpr int ROUTE_BUCKETS = 256;  // buckets of SCATTER, one per thread
static_assert(ROUTE_BUCKETS == EXT_THREADS, "a thread reserves its bucket's run");

// Dynamic shared memory of extract_kernel.
template <int NW, int MODE>
__host__ __device__ constexpr size_t extract_smem_bytes(uint32_t n_buckets) {
    if (MODE == HIST) return (size_t)n_buckets * 4;
    // u64 gdelta[256] | u32 hist[256] | u32 loff[256] | staged keys (u64 key,
    // u16 rank, u16 order) or positions (u16 rank, u16 order, u8 bucket)
    const size_t staged = NW == 1 ? (size_t)STAGE_KEYS * 12 : 0, byplace = (size_t)EXT_TILE * 5;
    return (size_t)ROUTE_BUCKETS * 16 + (staged > byplace ? staged : byplace);
}

// Inclusive scan of one value per thread over the CTA; *total = its sum.
// warp_sums: a buffer of its own per use (one barrier, no reuse).
__device__ __forceinline__ uint32_t tile_scan(uint32_t v, uint32_t* warp_sums, uint32_t* total) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += y;
    }
    if (lane == 31) warp_sums[warp] = v;
    __syncthreads();
    uint32_t before = 0, sum = 0;
#pragma unroll
    for (int w = 0; w < EXT_THREADS / 32; ++w) {
        const uint32_t t = warp_sums[w];
        before += w < warp ? t : 0u;
        sum += t;
    }
    *total = sum;
    return v + before;
}

template <int NW, int MODE>
__global__ void __launch_bounds__(EXT_THREADS, EXT_MIN_CTAS) extract_kernel(ExtractArgs a) {
    extern __shared__ __align__(16) uint8_t ext_smem[];
    __shared__ uint32_t sw[STREAM_WORDS];
    // emitting segments: emit mask << 32 | first arrival index << 8 | segment
    __shared__ uint64_t seg_list[EXT_THREADS];
    __shared__ uint32_t sums[3][EXT_THREADS / 32];
    __shared__ uint32_t hist_bases[MODE == HIST ? TILE_SEGS : 1];
    uint64_t* gdelta = reinterpret_cast<uint64_t*>(ext_smem);
    uint32_t* hist = MODE == HIST ? reinterpret_cast<uint32_t*>(ext_smem)
                                  : reinterpret_cast<uint32_t*>(gdelta + ROUTE_BUCKETS);
    uint32_t* loff = hist + ROUTE_BUCKETS;
    uint8_t* area = reinterpret_cast<uint8_t*>(loff + ROUTE_BUCKETS);
    // base bits of the segments: phase A only, in the staging area
    uint32_t* seg_bases = MODE == HIST ? hist_bases : reinterpret_cast<uint32_t*>(area);

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint64_t tile = a.tile_list ? (uint64_t)a.tile_list[blockIdx.x]
                                      : (uint64_t)blockIdx.x * (a.tile_stride > 1 ? a.tile_stride : 1u);
    uint64_t tile_start = tile * EXT_TILE;
    uint64_t n_end = a.n;
    bool halo_ok = tile_start > 0 || a.has_halo;
    uint32_t k = a.k;
    uint64_t bucket_off = 0;
    uint32_t set = 0;
    if (a.tiles) {
        const SetTile t = a.tiles[tile];
        tile_start = t.start;
        n_end = t.end;
        halo_ok = t.first_tile != tile;
        set = t.set;
        k = t.k;
        bucket_off = (uint64_t)t.set * a.n_buckets;
    }
    const uint64_t seg_start = tile_start + (uint64_t)tid * EXT_BPT;
    const uint32_t tile_line0 = (uint32_t)a.tile_line[tile];

    for (uint32_t b = tid; b < (MODE == HIST ? a.n_buckets : (uint32_t)ROUTE_BUCKETS); b += EXT_THREADS) hist[b] = 0;

    // ---- phase A: classify own segment (+ the halo segments)
    uint32_t w[8];
    const uint64_t valid = seg_start < n_end ? n_end - seg_start : 0;
    load32(a.buf + seg_start, valid, w);
    const Seg s = classify(w, valid);
    stream_put(sw, tid + HALO_SEGS, s.codes);
    seg_bases[tid + HALO_SEGS] = s.bases;
    if (tid < HALO_SEGS) {
        uint32_t hw[8];
        load32(a.buf + (int64_t)tile_start - HALO + 32 * tid, halo_ok ? 32 : 0, hw);
        const Seg h = classify(hw, halo_ok ? 32 : 0);
        stream_put(sw, tid, h.codes);
        seg_bases[tid] = h.bases;
    }
    if (tid < C_WORDS - 2 * TILE_SEGS) sw[2 * TILE_SEGS + tid] = 0;  // read past the last window, masked out
    uint32_t total;
    const uint32_t nl = (uint32_t)__popc(s.nls);
    const uint32_t line0 = tile_line0 + tile_scan(nl, sums[0], &total) - nl;  // the scan publishes seg_bases

    uint32_t emit = 0;
    const uint32_t seq = s.bases ? sequence_mask(line0, s.nls) : 0u;
    if (seq & s.bases) {
        const uint32_t* sb = seg_bases + tid + HALO_SEGS;  // sb[0] = this segment
        if constexpr (NW == 1) {
            emit = runs_at_least2(sb[-1], s.bases, k) & seq;
        } else if constexpr (NW == 4) {
            emit = runs_at_least5(sb[-4], sb[-3], sb[-2], sb[-1], s.bases, k) & seq;
        } else {
            const u128 X = ((u128)s.bases << 64) | ((u128)sb[-1] << 32) | (u128)sb[-2];
            emit = (uint32_t)(runs_at_least(X, k) >> 64) & seq;
        }
    }
    // k-mers (low half) and emitting segments (high half) up to this segment
    const uint32_t mine = (uint32_t)__popc(emit) | (emit ? 1u << 16 : 0u);
    const uint32_t upto = tile_scan(mine, sums[1], &total);
    const uint32_t n_tile = total & 0xFFFFu, n_segs = total >> 16;
    if (!n_tile) return;  // block-uniform: nothing to count in this tile (SCATTER reserves nothing)
    if (emit)
        seg_list[(upto >> 16) - 1] = ((uint64_t)emit << 32) | (((upto & 0xFFFFu) - (uint32_t)__popc(emit)) << 8) | (uint32_t)tid;
    __syncthreads();

    // ---- phase C
    const uint32_t lt = (1u << lane) - 1u;
    const uint32_t mask0 = key_mask(0, k);
    // lane `lane` of segment t: the window's place for t = 0 plus 2t words
    const StreamPos lane_pos = stream_pos((uint32_t)lane, k);
    auto pos_of = [&](uint32_t t) { return StreamPos{lane_pos.c + 2 * t, lane_pos.cs, lane_pos.f - 2 * t, lane_pos.fs}; };

    if constexpr (MODE == HIST) {
        const uint32_t shift = a.bucket_shift - 32;  // of the key's first 32 bits
        for (uint32_t i = warp; i < n_segs; i += EXT_THREADS / 32) {
            const uint64_t e = seg_list[i];
            if (((uint32_t)(e >> 32) >> lane) & 1u)
                atomicAdd(hist + (top_of_window(sw, pos_of((uint32_t)e & 0xFFu), mask0) >> shift), 1u);
        }
        __syncthreads();
        for (uint32_t b = tid; b < a.n_buckets; b += EXT_THREADS) {
            const uint32_t c = hist[b];
            if (c) atomicAdd(a.bucket_count + bucket_off + b, (unsigned long long)c);
        }
        return;
    }

    // Reserve bucket tid's run in the routed array, and the runs' offsets in
    // the tile's bucket order (loff): position p of that order, in bucket b,
    // belongs at routed[gdelta[b] + p].
    auto reserve = [&]() {
        const uint32_t c = hist[tid];
        const uint64_t rb = bucket_off + tid;  // the region (of this set)
        unsigned long long base = c ? atomicAdd(a.bucket_cursor + rb, (unsigned long long)c) : 0ull;
        if (a.region_end && c && base + c > a.region_end[rb]) {
            // the run does not fit the region: it goes whole to the
            // overflow area.  If that is full too, the batch is routed
            // again (error bit 1) and the run lands, in bounds, at the
            // overflow area's start (at least 65536 keys >= one run).
            atomicMin(a.region_fill + rb, base);
            // a multi-set batch has an overflow area per set
            unsigned long long* const ocur = a.set_ovf_cursor ? a.set_ovf_cursor + set : a.overflow_cursor;
            const uint64_t oend = a.set_ovf_cursor ? a.set_ovf_end[set] : a.overflow_end;
            const uint64_t ostart = a.set_ovf_cursor ? a.set_ovf_start[set] : a.overflow_start;
            const unsigned long long ob = atomicAdd(ocur, (unsigned long long)c);
            if (ob + c <= oend) {
                base = ob;
            } else {
                base = ostart;
                atomicOr(a.error, 2u);
            }
        }
        uint32_t sum;
        const uint32_t off = tile_scan(c, sums[2], &sum) - c;
        loff[tid] = off;
        gdelta[tid] = base - off;
        if (sum != n_tile) atomicOr(a.error, 1u);  // cannot happen: every listed k-mer was ranked once
        __syncthreads();
    };

    if (NW == 1 && n_tile <= (uint32_t)STAGE_KEYS) {
        uint64_t* skeys = reinterpret_cast<uint64_t*>(area);
        uint16_t* rank = reinterpret_cast<uint16_t*>(skeys + STAGE_KEYS);
        uint16_t* order = rank + STAGE_KEYS;
        const uint32_t mask1 = key_mask(1, k);
        for (uint32_t i = warp; i < n_segs; i += EXT_THREADS / 32) {
            const uint64_t e = seg_list[i];
            const uint32_t em = (uint32_t)(e >> 32);
            if (!((em >> lane) & 1u)) continue;
            const StreamPos p = pos_of((uint32_t)e & 0xFFu);
            const uint32_t f1 = sw[p.f + 1], c1 = sw[p.c + 1];
            const uint64_t F = ((uint64_t)funnel_l(sw[p.f], f1, p.fs) << 32) | funnel_l(f1, sw[p.f + 2], p.fs);
            const uint64_t C = ((uint64_t)funnel_l(sw[p.c], c1, p.cs) << 32) | funnel_l(c1, sw[p.c + 2], p.cs);
            const uint64_t key = (F < C ? F : C) & (((uint64_t)mask0 << 32) | mask1);
            const uint32_t arr = ((uint32_t)e >> 8) + (uint32_t)__popc(em & lt);  // < n_tile
            rank[arr] = (uint16_t)atomicAdd(hist + (uint32_t)(key >> 56), 1u);
            skeys[arr] = key;
        }
        __syncthreads();
        reserve();
        for (uint32_t i = tid; i < n_tile; i += EXT_THREADS)
            order[loff[(uint32_t)(skeys[i] >> 56)] + rank[i]] = (uint16_t)i;
        __syncthreads();
        uint64_t* out = reinterpret_cast<uint64_t*>(a.routed);
        for (uint32_t p = tid; p < n_tile; p += EXT_THREADS) {
            const uint64_t key = skeys[order[p]];
            out[gdelta[(uint32_t)(key >> 56)] + p] = key;
        }
        return;
    }

    {
        uint16_t* rank = reinterpret_cast<uint16_t*>(area);
        uint16_t* order = rank + EXT_TILE;
        uint8_t* bkt = reinterpret_cast<uint8_t*>(order + EXT_TILE);
        for (uint32_t i = warp; i < n_segs; i += EXT_THREADS / 32) {
            const uint64_t e = seg_list[i];
            if (!(((uint32_t)(e >> 32) >> lane) & 1u)) continue;
            const uint32_t t = (uint32_t)e & 0xFFu, at = 32 * t + lane;
            const uint32_t b = top_of_window(sw, pos_of(t), mask0) >> 24;
            rank[at] = (uint16_t)atomicAdd(hist + b, 1u);
            bkt[at] = (uint8_t)b;
        }
        __syncthreads();
        reserve();
        for (uint32_t i = warp; i < n_segs; i += EXT_THREADS / 32) {
            const uint64_t e = seg_list[i];
            if (!(((uint32_t)(e >> 32) >> lane) & 1u)) continue;
            const uint32_t at = 32 * ((uint32_t)e & 0xFFu) + lane;
            order[loff[bkt[at]] + rank[at]] = (uint16_t)at;
        }
        __syncthreads();
        for (uint32_t p = tid; p < n_tile; p += EXT_THREADS) {
            uint64_t key[NW];
            key_of_window<NW>(sw, stream_pos(order[p], k), k, key);
            const uint64_t at = gdelta[(uint32_t)(key[0] >> 56)] + p;
            if constexpr (NW == 1) {
                reinterpret_cast<uint64_t*>(a.routed)[at] = key[0];
            } else {
                ulonglong2* out = reinterpret_cast<ulonglong2*>(a.routed) + at * (NW / 2);
#pragma unroll
                for (int q = 0; q < NW / 2; ++q) out[q] = make_ulonglong2(key[2 * q], key[2 * q + 1]);
            }
        }
    }
}

// --------------------------------------------------- first occurrence + repeats

__device__ __forceinline__ uint64_t bloom_bits(uint64_t h) {
    // Three bit positions in one 64-bit word, taken from hash bits 40..57
    // (the word index uses the low bits).  The reference uses XXH3-128 and
    // (lo + i*(hi|1)) & 63 (src/BloomFilter.h:207-258); only the low/root
    // partition depends on this choice, never the merged counts.
    return (1ull << ((h >> 40) & 63)) | (1ull << ((h >> 46) & 63)) | (1ull << ((h >> 52) & 63));
}
// Three bit positions in a 32-bit filter word kept in a table cell (64-bit
// keys); hash bits 0..14, while the cell index uses bits 17 and up.
__device__ __forceinline__ uint32_t bloom_bits32(uint64_t h) {
    return (1u << (h & 31)) | (1u << ((h >> 5) & 31)) | (1u << ((h >> 10) & 31));
}

// Whether a cell reads empty (a 16-byte read may be torn while the cell is
// claimed: any EMPTY word counts as empty and is settled by the CAS), and
// whether it holds the key.
__device__ __forceinline__ bool cell_empty(uint64_t v) { return v == EMPTY; }
__device__ __forceinline__ bool cell_empty(const ulonglong2& v) { return v.x == EMPTY || v.y == EMPTY; }
__device__ __forceinline__ bool cell_holds(uint64_t v, uint64_t key) { return v == key; }
__device__ __forceinline__ bool cell_holds(const ulonglong2& v, const Key2& key) {
    return v.x == key.w0 && v.y == key.w1;
}
// Claim a 16-byte cell (or half of one) that read empty: its value after the
// CAS (the key's own when this thread claimed it).
__device__ __forceinline__ ulonglong2 claim16(void* s, const Key2& key) {
    const unsigned __int128 e = ~(unsigned __int128)0;
    const unsigned __int128 kv = ((unsigned __int128)key.w1 << 64) | key.w0;
    const unsigned __int128 old = atomicCAS(reinterpret_cast<unsigned __int128*>(s), e, kv);
    const unsigned __int128 now = old == e ? kv : old;
    return make_ulonglong2((uint64_t)now, (uint64_t)(now >> 64));
}

// Insert `add` occurrences of key into a bucket table starting at slot
// (h >> 17) & mask; false = probe limit hit.  Linear probing; a slot goes
// EMPTY -> key exactly once (CAS), counts only grow (atomicAdd).
static __device__ __noinline__ bool table_add_slow(Slot1* __restrict__ tab, uint64_t mask, uint64_t h, uint64_t key,
                                            uint32_t add, int first_p) {
    const uint64_t i = (h >> 17) & mask;
    const int limit = (int)min((uint64_t)PROBE_LIMIT, mask + 1);
    for (int p = first_p; p < limit; ++p) {
        Slot1* s = tab + ((i + p) & mask);
        uint64_t cur = __ldcg(&s->key);
        if (cur == EMPTY) {
            cur = atomicCAS(reinterpret_cast<unsigned long long*>(&s->key), EMPTY, key);
            if (cur == EMPTY) cur = key;
        }
        if (cur == key) {
            atomicAdd(&s->count, add);
            return true;
        }
    }
    return false;
}

static __device__ __noinline__ bool table_add_slow(Slot2* __restrict__ tab, uint64_t mask, uint64_t h, const Key2 key,
                                            uint32_t add, int first_p) {
    const uint64_t i = (h >> 17) & mask;
    const int limit = (int)min((uint64_t)PROBE_LIMIT, mask + 1);
    for (int p = first_p; p < limit; ++p) {
        Slot2* s = tab + ((i + p) & mask);
        const ulonglong2 v = __ldcg(reinterpret_cast<const ulonglong2*>(s));
        bool mine = (v.x == key.w0 && v.y == key.w1);
        // A 16-byte read that shows an EMPTY half may be torn, so ask the CAS
        // for the authoritative value.
        if (!mine && (v.x == EMPTY || v.y == EMPTY)) {
            const unsigned __int128 e = ~(unsigned __int128)0;
            const unsigned __int128 kv = ((unsigned __int128)key.w1 << 64) | key.w0;
            const unsigned __int128 old = atomicCAS(reinterpret_cast<unsigned __int128*>(s), e, kv);
            mine = (old == e) || (old == kv);
        }
        if (mine) {
            atomicAdd(&s->count, add);
            return true;
        }
    }
    return false;
}

__device__ __forceinline__ bool same_key(uint64_t a, uint64_t b) { return a == b; }
__device__ __forceinline__ bool same_key(const Key2& a, const Key2& b) { return a.w0 == b.w0 && a.w1 == b.w1; }
KC_HD bool same_key(const Key4& a, const Key4& b) {
    return a.w0 == b.w0 && a.w1 == b.w1 && a.w2 == b.w2 && a.w3 == b.w3;
}
// Whether a slot read without a fence while its key may be arriving holds
// `key`: every word was EMPTY before it was written, once, so a read that
// agrees in all words holds no unwritten one, unless the key itself has a word
// of all ones (32 T's in its place).
KC_HD bool holds_unfenced(const Key4& have, const Key4& key) {
    return same_key(have, key) && key.w0 != EMPTY && key.w1 != EMPTY && key.w2 != EMPTY && key.w3 != EMPTY;
}
__device__ __forceinline__ Key4 cell_key4(const Slot4* s) {
    const ulonglong2 a = __ldcg(reinterpret_cast<const ulonglong2*>(s));
    const ulonglong2 b = __ldcg(reinterpret_cast<const ulonglong2*>(s) + 1);
    return Key4{a.x, a.y, b.x, b.y};
}

// Insert `add` occurrences of a 256-bit key, probing from (h >> 17) & mask.
// Returns 1 when added, 0 when the probe limit was hit (the bucket
// overflows; or `overflowed` says that it has), -1 when a slot stayed
// SLOT_WRITING for PUBLISH_WAIT_LIMIT polls.
static __device__ __noinline__ int table_add4(Slot4* __restrict__ tab, uint64_t mask, uint64_t h, const Key4& key,
                                              uint32_t add, const uint32_t* overflowed) {
    const uint64_t i = (h >> 17) & mask;
    const int limit = (int)min((uint64_t)PROBE_LIMIT, mask + 1);
    for (int p = 0; p < limit; ++p) {
        if (p && p % PROBE_CHECK == 0 && overflowed && __ldcg(overflowed)) return 0;
        Slot4* s = tab + ((i + p) & mask);
        volatile uint32_t* state = &s->state;
        // state and key in one round trip, with nothing that orders the two:
        // the key words of a READY slot may still be the unwritten ones.  A
        // match that cannot mix the two counts (holds_unfenced); anything else
        // is read again behind a fence.  A fence per probe and a second round
        // trip made the count of 136 M keys (k = 101, counted here) 7.56 ms,
        // 6.62 so.
        uint32_t st = *state;
        Key4 have = cell_key4(s);
        if (st == SLOT_READY && holds_unfenced(have, key)) {
            atomicAdd(&s->count, add);
            return 1;
        }
        if (st == SLOT_EMPTY) {
            st = atomicCAS(&s->state, SLOT_EMPTY, SLOT_WRITING);
            if (st == SLOT_EMPTY) {  // claimed: key and first count, then publish
                s->w0 = key.w0;
                s->w1 = key.w1;
                s->w2 = key.w2;
                s->w3 = key.w3;
                s->count = add;
                __threadfence();
                atomicExch(&s->state, SLOT_READY);
                return 1;
            }
        }
        for (uint32_t n = 0; st == SLOT_WRITING; ++n) {
            if (n >= PUBLISH_WAIT_LIMIT) return -1;
            st = *state;
        }
        __threadfence();  // pairs with the owner's fence: its key words are visible
        have = cell_key4(s);
        if (same_key(have, key)) {
            atomicAdd(&s->count, add);
            return 1;
        }
    }
    return 0;
}

// The same for k <= 127, where neither 16-byte half of a canonical key is all
// ones (its first half would take 64 T in one orientation and 64 A in the
// other, its last ends in unused zero bits): a slot is claimed half by half,
// each with one 16-byte CAS.  The first half decides who may claim the second,
// the second whose slot it is; a key that loses the second goes on to the next
// slot.  No fence and no wait, of which the published state cost every warp
// several in turn: 136 M keys of k = 101 counted in 3.74 ms, 6.59 before (the
// table cell read beside the filter word as for shorter keys: no gain).
// false = probe limit hit, or `overflowed` says that the bucket has.
__device__ __forceinline__ bool table_add4_halves(Slot4* __restrict__ tab, uint64_t mask, uint64_t h, const Key4& key,
                                                  uint32_t add, const uint32_t* overflowed) {
    const uint64_t i = (h >> 17) & mask;
    const uint32_t limit = (uint32_t)min((uint64_t)PROBE_LIMIT, mask + 1);
    const Key2 k0{key.w0, key.w1}, k1{key.w2, key.w3};
    for (uint32_t p = 0; p < limit; ++p) {
        if (p && p % PROBE_CHECK == 0 && __ldcg(overflowed)) return false;
        Slot4* s = tab + ((i + p) & mask);
        ulonglong2* halves = reinterpret_cast<ulonglong2*>(s);
        ulonglong2 a = __ldcg(halves), b = __ldcg(halves + 1);
        // (a half that shows an EMPTY word may be torn: the CAS tells)
        if (cell_empty(a)) a = claim16(halves, k0);
        if (!cell_holds(a, k0)) continue;
        if (cell_empty(b)) {
            b = claim16(halves + 1, k1);
            if (cell_holds(b, k1)) s->state = SLOT_READY;  // (all that get here store the same)
        }
        if (!cell_holds(b, k1)) continue;
        atomicAdd(&s->count, add);
        return true;
    }
    return false;
}

// Full insert (used by the table rehash).
__device__ __forceinline__ bool table_add(Slot1* tab, uint64_t mask, uint64_t h, uint64_t key, uint32_t add) {
    return table_add_slow(tab, mask, h, key, add, 0);
}
__device__ __forceinline__ bool table_add(Slot2* tab, uint64_t mask, uint64_t h, const Key2& key, uint32_t add) {
    return table_add_slow(tab, mask, h, key, add, 0);
}
__device__ __forceinline__ bool table_add(Slot4* tab, uint64_t mask, uint64_t h, const Key4& key, uint32_t add) {
    return table_add4(tab, mask, h, key, add, nullptr) > 0;
}

// Probe-round helpers of count_routed (64- and 128-bit keys): a cell's key
// as read, and the claim of a cell read empty (returns the cell's key after
// the CAS: `key` when this thread claimed it).
__device__ __forceinline__ uint64_t read_cell(const Slot1* s) { return __ldcg(&s->key); }
__device__ __forceinline__ ulonglong2 read_cell(const Slot2* s) {
    return __ldcg(reinterpret_cast<const ulonglong2*>(s));
}
__device__ __forceinline__ uint64_t claim_cell(Slot1* s, uint64_t key) {
    const uint64_t old = atomicCAS(reinterpret_cast<unsigned long long*>(&s->key), EMPTY, key);
    return old == EMPTY ? key : old;
}
__device__ __forceinline__ ulonglong2 claim_cell(Slot2* s, const Key2& key) { return claim16(s, key); }

__device__ __forceinline__ uint64_t key_of_lane(uint64_t k, int lane) { return __shfl_sync(0xffffffffu, k, lane); }
__device__ __forceinline__ Key2 key_of_lane(const Key2& k, int lane) {
    return Key2{__shfl_sync(0xffffffffu, k.w0, lane), __shfl_sync(0xffffffffu, k.w1, lane)};
}

// Keys with long probe sequences: the n keys before `end` (a segment's back),
// whose first PROBE_CHECK cells hold other keys, are inserted one after another
// by the whole warp, 32 cells a round, of which those that hold the key or read
// empty are settled in probe order.  Keys that find no room in their probe
// window, or whose bucket has overflowed already, stay; returns their number.
template <class S, class K>
static __device__ __forceinline__ uint32_t insert_far(K* end, uint32_t n, uint32_t bucket0, S* __restrict__ table,
                                                   const BucketMeta* __restrict__ meta, uint32_t bucket_shift,
                                                   uint32_t* bucket_overflow) {
    const uint32_t lane = threadIdx.x & 31;
    uint32_t kept = 0;
    for (uint32_t i0 = 0; i0 < n; i0 += 32) {
        const bool in = i0 + lane < n;
        K own = *(end - 1 - (in ? i0 + lane : i0));
        __syncwarp();  // every read precedes the writes below
        uint32_t failed = 0;
        for (uint32_t left = __ballot_sync(0xffffffffu, in); left;) {
            const K key = key_of_lane(own, __ffs(left) - 1);
            const uint32_t same = __ballot_sync(0xffffffffu, in && same_key(own, key));  // its occurrences
            left &= ~same;
            const uint32_t b = bucket0 + (uint32_t)(key_hi(key) >> bucket_shift);
            S* tab = table + __ldg(&meta[b].tab_off);
            const uint32_t mask = (uint32_t)__ldg(&meta[b].tab_mask);
            const uint32_t limit = (uint32_t)min((uint64_t)PROBE_LIMIT, (uint64_t)mask + 1);
            const uint32_t home = (uint32_t)(hash_key(key) >> 17);
            bool added = false;
            const bool full = __ldcg(bucket_overflow + b) != 0;
            if (__any_sync(0xffffffffu, full)) {
                failed |= same;
                continue;
            }
            for (uint32_t p = PROBE_CHECK; p < limit && !added; p += 32) {
                S* s = tab + ((home + p + lane) & mask);
                auto v = read_cell(s);
                uint32_t open = __ballot_sync(0xffffffffu, p + lane < limit && (cell_empty(v) || cell_holds(v, key)));
                for (; open && !added; open &= open - 1) {
                    bool mine = false;
                    if (lane == __ffs(open) - 1) {
                        if (cell_empty(v)) v = claim_cell(s, key);
                        mine = cell_holds(v, key);
                        if (mine) atomicAdd(&s->count, (uint32_t)__popc(same));
                    }
                    added = __any_sync(0xffffffffu, mine);
                }
            }
            if (!added) {
                failed |= same;
                if (lane == 0) bucket_overflow[b] = 1u;
            }
        }
        if ((failed >> lane) & 1u) *(end - 1 - (kept + __popc(failed & ((1u << lane) - 1u)))) = own;
        kept += __popc(failed);
        __syncwarp();
    }
    return kept;
}

template <int NW>
struct SlotOf;
template <>
struct SlotOf<1> {
    using T = Slot1;
};
template <>
struct SlotOf<2> {
    using T = Slot2;
};
template <>
struct SlotOf<4> {
    using T = Slot4;
};

// Keys per lane of the count kernel and its CTAs per SM (the register budget
// is 65536 / (256 x CTAs)).  The kernel waits on L2 round trips, so resident
// warps hide more than items per lane: for 64-bit keys 2 items at 6 CTAs/SM
// (40 registers) ran 42.7 ms where 4 items at 4 CTAs ran 47.4 and 6 at 3 ran
// 58.3 (genome-scale step, same counts); for 128-bit keys 2 items at 4 CTAs
// ran 233 ms where 5 CTAs (48 registers) ran 246 (the full k=63 shape, ten
// passes over 48 GB of tables; at a tenth of that size 5 CTAs were ahead).
template <int NW>
__host__ __device__ constexpr int count_items() {
    return NW == 1 ? 2 : (NW == 2 ? 2 : 1);
}
template <int NW, bool HALVES = false>
__host__ __device__ constexpr int count_min_ctas() {
    return NW == 1 ? 6 : (NW == 2 ? 4 : (HALVES ? 6 : 4));
}
// Keys owned by one warp of the count kernel (a contiguous segment).
template <int NW>
__host__ __device__ constexpr int count_seg() {
    return 32 * count_items<NW>();
}
template <int NW>
__host__ __device__ constexpr int count_tile() {
    return CNT_THREADS * count_items<NW>();
}

struct CountArgs {
    void* routed;                 // bucket-contiguous keys of this batch
    uint64_t n_keys;
    const BucketMeta* meta;
    uint64_t* bloom;
    void* table;
    uint32_t* seg_low;            // per warp segment: first occurrences kept at its front
    uint32_t* seg_fail;           // per warp segment: overflowed keys kept at its back
    uint32_t* bucket_overflow;    // set to 1 for a bucket whose table overflowed
    uint32_t* error;              // 256-bit keys: set when a slot was never published
    uint32_t bucket_shift;
    uint32_t n_buckets;
    int use_filter;               // 0: retry pass (table only, no filter)
    // 64-bit keys: the filter words are the pad fields of table cells
    // (bloom_off / bloom_mask count cells of the table arena)
    uint32_t filter_in_table;
    // multi-set batch: set s owns segments [set_seg_start[s], set_seg_start[s+1])
    // and buckets [s * set_buckets, (s + 1) * set_buckets); EMPTY keys are gaps
    const uint64_t* set_seg_start;
    uint32_t n_sets;
    uint32_t set_buckets;
};

// Bucket placement as read by the count kernel (shared memory copy).
struct MetaS {
    uint64_t bloom_off, tab_off;
    uint32_t bloom_mask, tab_mask;
};
constexpr int META_SMEM_BUCKETS = 256;
constexpr int CNT_SEGS_PER_WARP = 8;

// For each routed key: the first-occurrence filter decides low.bin (first)
// or the repeat table (seen before), as the reference's classifier does with
// ConcurrentBloomFilter::insert (src/FastqClassifier.h:241-349,
// src/BloomFilter.h:207-234): a relaxed read first, then fetch_or; "first" =
// the old word lacked one of the bits.  Repeats increment the bucket's
// open-addressing table (replaces KmerTree + ConcurrentMap::increment,
// src/NewKmerTree.h:383-489, src/ConcurrentMap.h:112-160).
//
// Persistent CTAs; each warp walks contiguous segments of count_seg<NW>()
// keys.  Per segment: equal keys inside the warp are merged
// (__match_any_sync); every item's filter word and first table slot are read
// together (one round trip settles most repeats); filter atomics and table
// adds follow.  Outputs are compacted IN PLACE into the warp's own segment
// (only this warp reads it; __syncwarp orders reads before writes): first
// occurrences at the front, keys that met a full table at the back.
// CELLS2: 128-bit keys whose filter words are fields of the table cells (a run
// counted in windows; its spilled, retried and later keys come here).
// HALVES: 256-bit keys of k <= 127 (table_add4_halves).
template <int NW, bool CELLS2 = false, bool HALVES = false>
__global__ void __launch_bounds__(CNT_THREADS, count_min_ctas<NW, HALVES>()) count_routed(CountArgs a) {
    static_assert(!CELLS2 || NW == 2, "128-bit keys only");
    static_assert(!HALVES || NW == 4, "256-bit keys only");
    using K = typename KeyOf<NW>::T;
    using S = typename SlotOf<NW>::T;
    // first table slot read ahead of the filter result (not for 256-bit keys,
    // whose slots are read under the publish protocol of table_add4)
    using Seen = typename std::conditional<NW == 1, uint64_t,
                                           typename std::conditional<NW == 2, ulonglong2, uint32_t>::type>::type;
    constexpr int ITEMS = count_items<NW>();
    constexpr int SEG = count_seg<NW>();
    __shared__ MetaS sm[META_SMEM_BUCKETS];
    const bool meta_in_smem = a.n_buckets <= META_SMEM_BUCKETS;
    if (meta_in_smem) {
        for (uint32_t b = threadIdx.x; b < a.n_buckets; b += blockDim.x) {
            const BucketMeta m = a.meta[b];
            sm[b] = MetaS{m.bloom_off, m.tab_off, (uint32_t)m.bloom_mask, (uint32_t)m.tab_mask};
        }
        __syncthreads();
    }
    auto meta_of = [&](uint32_t b) -> MetaS {
        if (meta_in_smem) return sm[b];
        const BucketMeta* m = a.meta + b;
        return MetaS{__ldg(&m->bloom_off), __ldg(&m->tab_off), (uint32_t)__ldg(&m->bloom_mask),
                     (uint32_t)__ldg(&m->tab_mask)};
    };

    K* keys = reinterpret_cast<K*>(a.routed);
    S* table = reinterpret_cast<S*>(a.table);
    const int lane = threadIdx.x & 31;
    const uint32_t lt = (1u << lane) - 1u;
    const uint64_t n_segs = (a.n_keys + SEG - 1) / SEG;
    // Each CTA owns CNT_SEGS_PER_WARP consecutive segments per warp; CTAs are
    // dispatched in blockIdx order, so the keys in flight stay within a narrow
    // window of the bucket-sorted array (one or two buckets' filter and table
    // lines live in L2 at a time).
    auto bucket0_of = [&](uint64_t gw) {  // first bucket of the set that segment gw belongs to
        if (!a.n_sets) return 0u;
        uint32_t lo = 0, hi = a.n_sets;  // last set whose first segment <= gw
        while (hi - lo > 1) {
            const uint32_t mid = (lo + hi) / 2;
            if (a.set_seg_start[mid] <= gw) lo = mid;
            else hi = mid;
        }
        return lo * a.set_buckets;
    };
    __shared__ uint32_t s_far[CNT_THREADS / 32];  // keys lie at the back of some of the warp's segments
    if (NW <= 2 && lane == 0) s_far[threadIdx.x >> 5] = 0;
    const uint64_t cta_seg0 = (uint64_t)blockIdx.x * (CNT_THREADS / 32) * CNT_SEGS_PER_WARP;
    const uint64_t cta_seg1 = min(n_segs, cta_seg0 + (uint64_t)(CNT_THREADS / 32) * CNT_SEGS_PER_WARP);
    for (uint64_t gw = cta_seg0 + (threadIdx.x >> 5); gw < cta_seg1; gw += CNT_THREADS / 32) {
        const uint64_t s0 = gw * SEG;
        const uint64_t s_end = min(a.n_keys, s0 + SEG);
        uint64_t base = s0;
        uint32_t n_in = (uint32_t)(s_end - s0);
        if (!a.use_filter) {
            const uint32_t nf = a.seg_fail[gw];
            if (nf == 0) continue;  // warp-uniform
            base = s_end - nf;
            n_in = nf;
        }

        const uint32_t set_bucket0 = bucket0_of(gw);
        K it[ITEMS];
        uint32_t mult[ITEMS];
#pragma unroll
        for (int j = 0; j < ITEMS; ++j) {
            const uint32_t idx = (uint32_t)(j * 32 + lane);
            mult[j] = idx < n_in ? 1u : 0u;
            if constexpr (NW == 1) it[j] = EMPTY;
            else if constexpr (NW == 2) it[j] = Key2{EMPTY, EMPTY};
            else it[j] = Key4{EMPTY, EMPTY, EMPTY, EMPTY};
            if (mult[j]) {
                it[j] = keys[base + idx];
                if constexpr (NW == 1) mult[j] = it[j] != EMPTY;
                else if constexpr (NW == 2) mult[j] = !(it[j].w0 == EMPTY && it[j].w1 == EMPTY);
                else mult[j] = !(it[j].w0 == EMPTY && it[j].w1 == EMPTY && it[j].w2 == EMPTY && it[j].w3 == EMPTY);
            }
        }
        __syncwarp();  // every read of the segment precedes any in-place write

        // merge equal keys: the lowest lane of a group carries the multiplicity.
        // Equal keys inside one segment arrive in runs (a hot k-mer repeated
        // along a read lands in consecutive routed slots), so the full match
        // runs only when some lane's key equals its neighbour's; otherwise the
        // warp goes on with one atomic per key, which is exact either way.
#pragma unroll
        for (int j = 0; j < ITEMS; ++j) {
            bool eq_next;
            if constexpr (NW == 1) {
                const uint64_t nx = __shfl_down_sync(0xffffffffu, it[j], 1);
                eq_next = nx == it[j];
            } else if constexpr (NW == 2) {
                const uint64_t n0 = __shfl_down_sync(0xffffffffu, it[j].w0, 1);
                const uint64_t n1 = __shfl_down_sync(0xffffffffu, it[j].w1, 1);
                eq_next = n0 == it[j].w0 && n1 == it[j].w1;
            } else {
                const uint64_t n0 = __shfl_down_sync(0xffffffffu, it[j].w0, 1);
                const uint64_t n1 = __shfl_down_sync(0xffffffffu, it[j].w1, 1);
                const uint64_t n2 = __shfl_down_sync(0xffffffffu, it[j].w2, 1);
                const uint64_t n3 = __shfl_down_sync(0xffffffffu, it[j].w3, 1);
                eq_next = n0 == it[j].w0 && n1 == it[j].w1 && n2 == it[j].w2 && n3 == it[j].w3;
            }
            if (!__any_sync(0xffffffffu, eq_next && lane < 31 && mult[j] != 0)) continue;  // warp-uniform
            const uint32_t active = __ballot_sync(0xffffffffu, mult[j] != 0);
            if (mult[j]) {
                uint32_t same;
                if constexpr (NW == 1) same = __match_any_sync(active, it[j]);
                else if constexpr (NW == 2) same = __match_any_sync(active, it[j].w0) & __match_any_sync(active, it[j].w1);
                else
                    same = __match_any_sync(active, it[j].w0) & __match_any_sync(active, it[j].w1) &
                           __match_any_sync(active, it[j].w2) & __match_any_sync(active, it[j].w3);
                mult[j] = ((__ffs(same) - 1) == lane) ? (uint32_t)__popc(same) : 0u;
            }
        }

        // one round trip: filter word + first table slot of every item
        uint64_t h[ITEMS];
        uint64_t old[ITEMS];
        Seen seen[ITEMS];
#pragma unroll
        for (int j = 0; j < ITEMS; ++j) {
            if (mult[j]) {
                h[j] = hash_key(it[j]);
                const MetaS m = meta_of(set_bucket0 + (uint32_t)(key_hi(it[j]) >> a.bucket_shift));
                const S* slot = table + m.tab_off + ((h[j] >> 17) & m.tab_mask);
                if constexpr (NW == 1) {
                    if (a.filter_in_table) {
                        // the filter word is the cell's pad field, at the index
                        // of the first table probe: one 16-byte read gives key,
                        // count and filter bits unless the bucket's table has
                        // moved to a grown region (then the cells are filter only)
                        const ulonglong2 cv = __ldcg(reinterpret_cast<const ulonglong2*>(
                            table + m.bloom_off + ((h[j] >> 17) & m.bloom_mask)));
                        old[j] = cv.y >> 32;
                        seen[j] = m.bloom_off == m.tab_off ? cv.x : __ldcg(&slot->key);
                    } else {
                        if (a.use_filter) old[j] = __ldcg(a.bloom + m.bloom_off + (h[j] & m.bloom_mask));
                        seen[j] = __ldcg(&slot->key);
                    }
                } else {
                    if constexpr (CELLS2)
                        old[j] = __ldcg(&(table + m.bloom_off + ((h[j] >> 17) & m.bloom_mask))->pad[0]);
                    else if (a.use_filter)
                        old[j] = __ldcg(a.bloom + m.bloom_off + (h[j] & m.bloom_mask));
                    if constexpr (NW == 2) seen[j] = __ldcg(reinterpret_cast<const ulonglong2*>(slot));
                    else seen[j] = 0;
                }
            }
        }
        uint32_t first_bits = 0;  // bit j: item j is a first occurrence
        if (a.use_filter) {
            // every item's filter atomic is issued before any old value is
            // tested (old[j] is replaced by the atomic's return value; an item
            // whose bits were all set already keeps its read value)
            bool in_table = CELLS2;
            if constexpr (NW == 1) in_table = a.filter_in_table != 0;
            uint32_t issued = 0;
#pragma unroll
            for (int j = 0; j < ITEMS; ++j) {
                if (mult[j]) {
                    const uint64_t bits = in_table ? (uint64_t)bloom_bits32(h[j]) : bloom_bits(h[j]);
                    if ((old[j] & bits) != bits) {
                        const MetaS m = meta_of(set_bucket0 + (uint32_t)(key_hi(it[j]) >> a.bucket_shift));
                        if constexpr (NW == 1) {
                            if (in_table)
                                old[j] = atomicOr(&(table + m.bloom_off + ((h[j] >> 17) & m.bloom_mask))->pad,
                                                  (uint32_t)bits);
                            else
                                old[j] = atomicOr(reinterpret_cast<unsigned long long*>(a.bloom + m.bloom_off +
                                                                                        (h[j] & m.bloom_mask)),
                                                  bits);
                        } else if constexpr (CELLS2) {
                            old[j] = atomicOr(&(table + m.bloom_off + ((h[j] >> 17) & m.bloom_mask))->pad[0],
                                              (uint32_t)bits);
                        } else {
                            old[j] = atomicOr(
                                reinterpret_cast<unsigned long long*>(a.bloom + m.bloom_off + (h[j] & m.bloom_mask)), bits);
                        }
                        issued |= 1u << j;
                    }
                }
            }
#pragma unroll
            for (int j = 0; j < ITEMS; ++j) {
                if ((issued >> j) & 1u) {
                    const uint64_t bits = in_table ? (uint64_t)bloom_bits32(h[j]) : bloom_bits(h[j]);
                    if ((old[j] & bits) != bits) first_bits |= 1u << j;
                }
            }
        }
        uint32_t fail_bits = 0;
        if constexpr (NW == 4) {
#pragma unroll
            for (int j = 0; j < ITEMS; ++j) {
                const uint32_t reps = mult[j] - ((first_bits >> j) & 1u);
                if (mult[j] && reps) {
                    const uint32_t b = set_bucket0 + (uint32_t)(key_hi(it[j]) >> a.bucket_shift);
                    const MetaS m = meta_of(b);
                    int r;
                    if constexpr (HALVES)
                        r = table_add4_halves(table + m.tab_off, m.tab_mask, h[j], it[j], reps, a.bucket_overflow + b);
                    else r = table_add4(table + m.tab_off, m.tab_mask, h[j], it[j], reps, a.bucket_overflow + b);
                    if (r < 0) atomicOr(a.error, 1u);  // a slot was never published: reported, not retried
                    if (r == 0) {
                        fail_bits |= 1u << j;
                        mult[j] = reps;  // keep the count that still has to be added
                        a.bucket_overflow[b] = 1u;
                    }
                }
            }
        } else {
            // Repeats into the table by linear probing in lockstep rounds.
            // Round p settles every item whose probe cell p it has read
            // (`seen`; round 0 is the cell read with the filter word): the
            // claims of all items (CAS on a cell read EMPTY, or with an EMPTY
            // half for 128-bit keys) are issued before any result is used,
            // then items whose cell holds their key add their count, and items
            // that met another key read their next cell together.  A collision
            // in one lane costs the warp one more round for all its items,
            // not one more dependent chain per item.
            uint32_t todo = 0;
#pragma unroll
            for (int j = 0; j < ITEMS; ++j) {
                mult[j] = mult[j] ? mult[j] - ((first_bits >> j) & 1u) : 0u;  // occurrences left to add
                if (mult[j]) todo |= 1u << j;
            }
            for (uint32_t p = 0;; ++p) {
#pragma unroll
                for (int j = 0; j < ITEMS; ++j) {
                    if (((todo >> j) & 1u) && cell_empty(seen[j])) {
                        const MetaS m = meta_of(set_bucket0 + (uint32_t)(key_hi(it[j]) >> a.bucket_shift));
                        seen[j] = claim_cell(table + m.tab_off + (((h[j] >> 17) + p) & m.tab_mask), it[j]);
                    }
                }
#pragma unroll
                for (int j = 0; j < ITEMS; ++j) {
                    if (!((todo >> j) & 1u)) continue;
                    const uint32_t b = set_bucket0 + (uint32_t)(key_hi(it[j]) >> a.bucket_shift);
                    const MetaS m = meta_of(b);
                    if (cell_holds(seen[j], it[j])) {
                        atomicAdd(&table[m.tab_off + (((h[j] >> 17) + p) & m.tab_mask)].count, mult[j]);
                        todo &= ~(1u << j);
                    } else if ((uint64_t)p + 1 >= min((uint64_t)PROBE_LIMIT, (uint64_t)m.tab_mask + 1)) {
                        fail_bits |= 1u << j;  // mult[j] keeps the count that still has to be added
                        todo &= ~(1u << j);
                        a.bucket_overflow[b] = 1u;
                    }
                }
                if (!__any_sync(0xffffffffu, todo != 0)) break;  // warp-uniform
                if (p + 1 == PROBE_CHECK) {  // the rest by insert_far
                    fail_bits |= todo;
                    break;
                }
#pragma unroll
                for (int j = 0; j < ITEMS; ++j) {
                    if ((todo >> j) & 1u) {
                        const MetaS m = meta_of(set_bucket0 + (uint32_t)(key_hi(it[j]) >> a.bucket_shift));
                        seen[j] = read_cell(table + m.tab_off + (((h[j] >> 17) + p + 1) & m.tab_mask));
                    }
                }
            }
        }

        // in-place compaction inside the warp's segment
        uint32_t n_low = 0, n_fail = 0;
#pragma unroll
        for (int j = 0; j < ITEMS; ++j) {
            const bool first = (first_bits >> j) & 1u;
            const uint32_t lm = __ballot_sync(0xffffffffu, first);
            if (first) keys[s0 + n_low + __popc(lm & lt)] = it[j];
            n_low += __popc(lm);
        }
        if (__any_sync(0xffffffffu, fail_bits != 0)) {
#pragma unroll
            for (int j = 0; j < ITEMS; ++j) {
                const uint32_t f = ((fail_bits >> j) & 1u) ? mult[j] : 0u;
                uint32_t fsum = f;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const uint32_t y = __shfl_up_sync(0xffffffffu, fsum, o);
                    if (lane >= o) fsum += y;
                }
                const uint32_t wtot = __shfl_sync(0xffffffffu, fsum, 31);
                const uint32_t my0 = n_fail + fsum - f;
                for (uint32_t r = 0; r < f; ++r) keys[s_end - 1 - (my0 + r)] = it[j];
                n_fail += wtot;
            }
            if (NW <= 2 && lane == 0) s_far[threadIdx.x >> 5] = 1;
        }
        if (lane == 0) {
            if (a.use_filter) a.seg_low[gw] = n_low;
            a.seg_fail[gw] = n_fail;
        }
    }
    // Long probe sequences, once the warp's segments are through: looked into
    // in the rounds above they cost the kernel 200 bytes of spills (10 M reads
    // in five passes, 64-bit keys: count 4.6 ms without, 6.5 with).
    if constexpr (NW <= 2) {
        __syncwarp();
        if (!s_far[threadIdx.x >> 5]) return;
        for (uint64_t gw = cta_seg0 + (threadIdx.x >> 5); gw < cta_seg1; gw += CNT_THREADS / 32) {
            const uint32_t nf = a.seg_fail[gw];
            if (nf == 0) continue;  // warp-uniform
            const uint32_t kept = insert_far(keys + min(a.n_keys, gw * SEG + SEG), nf, bucket0_of(gw), table, a.meta,
                                             a.bucket_shift, a.bucket_overflow);
            if (lane == 0) a.seg_fail[gw] = kept;
        }
    }
}

// Move every occupied slot of one bucket's old table into its new table.
template <int NW>
__global__ void rehash_bucket(const void* old_tab, uint64_t old_slots, void* new_tab, uint64_t new_mask,
                              uint32_t* failed) {
    using S = typename SlotOf<NW>::T;
    const S* src = reinterpret_cast<const S*>(old_tab);
    S* dst = reinterpret_cast<S*>(new_tab);
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < old_slots;
         i += (uint64_t)gridDim.x * blockDim.x) {
        const S s = src[i];
        if constexpr (NW == 1) {
            if (s.key == EMPTY) continue;
            if (!table_add(dst, new_mask, hash_key(s.key), s.key, s.count)) atomicExch(failed, 1u);
        } else if constexpr (NW == 2) {
            if (s.w0 == EMPTY && s.w1 == EMPTY) continue;
            const Key2 k{s.w0, s.w1};
            if (!table_add(dst, new_mask, hash_key(k), k, s.count)) atomicExch(failed, 1u);
        } else {
            if (s.state != SLOT_READY) continue;
            const Key4 k{s.w0, s.w1, s.w2, s.w3};
            if (!table_add(dst, new_mask, hash_key(k), k, s.count)) atomicExch(failed, 1u);
        }
    }
}

// One bucket's table growth: its old table (old_off, old_slots slots) moves
// into a new table of new_mask + 1 slots at new_off (slot offsets in the
// table arena).
struct GrowJob {
    uint64_t old_off, old_slots, new_off, new_mask;
};

template <int NW>
__device__ __forceinline__ void init_slot(typename SlotOf<NW>::T& s) {
    if constexpr (NW == 1) {
        s.key = EMPTY;
        s.count = 0;
        s.pad = 0;
    } else if constexpr (NW == 2) {
        s.w0 = EMPTY;
        s.w1 = EMPTY;
        s.count = 0;
        s.pad[0] = s.pad[1] = s.pad[2] = 0;
    } else {
        s.w0 = s.w1 = s.w2 = s.w3 = EMPTY;
        s.count = 0;
        s.state = SLOT_EMPTY;
        s.mark = 0;
    }
}

// Many growths at once: blockIdx.y = job; the new tables are initialised by
// grow_init, then grow_move moves every occupied old slot (failed[job] = 1
// when a key met a full probe window of the new table).
template <int NW>
__global__ void grow_init(void* table, const GrowJob* __restrict__ jobs) {
    using S = typename SlotOf<NW>::T;
    const GrowJob j = jobs[blockIdx.y];
    S* t = reinterpret_cast<S*>(table) + j.new_off;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i <= j.new_mask;
         i += (uint64_t)gridDim.x * blockDim.x) {
        S s;
        init_slot<NW>(s);
        t[i] = s;
    }
}

template <int NW>
__global__ void grow_move(void* table, const GrowJob* __restrict__ jobs, uint32_t* __restrict__ failed) {
    using S = typename SlotOf<NW>::T;
    const GrowJob j = jobs[blockIdx.y];
    const S* src = reinterpret_cast<const S*>(table) + j.old_off;
    S* dst = reinterpret_cast<S*>(table) + j.new_off;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < j.old_slots;
         i += (uint64_t)gridDim.x * blockDim.x) {
        const S s = src[i];
        if constexpr (NW == 1) {
            if (s.key == EMPTY) continue;
            if (!table_add(dst, j.new_mask, hash_key(s.key), s.key, s.count)) failed[blockIdx.y] = 1u;
        } else if constexpr (NW == 2) {
            if (s.w0 == EMPTY && s.w1 == EMPTY) continue;
            const Key2 k{s.w0, s.w1};
            if (!table_add(dst, j.new_mask, hash_key(k), k, s.count)) failed[blockIdx.y] = 1u;
        } else {
            if (s.state != SLOT_READY) continue;
            const Key4 k{s.w0, s.w1, s.w2, s.w3};
            if (!table_add(dst, j.new_mask, hash_key(k), k, s.count)) failed[blockIdx.y] = 1u;
        }
    }
}

// Initialise table slots to EMPTY with count 0.
template <int NW>
__global__ void init_slots(void* tab, uint64_t n) {
    // the table as 16-byte words, each lane one coalesced word per step: a
    // slot is 1, 2 or 3 words, EMPTY keys are all ones, counts, padding,
    // the 256-bit slot's state (SLOT_EMPTY = 0) and mark are zeros
    using S = typename SlotOf<NW>::T;
    constexpr uint64_t Q = sizeof(S) / 16;
    static_assert(sizeof(S) % 16 == 0, "slots are whole 16-byte words");
    uint4* t = reinterpret_cast<uint4*>(tab);
    const uint64_t n16 = n * Q;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n16; i += (uint64_t)gridDim.x * blockDim.x) {
        uint4 v = make_uint4(0u, 0u, 0u, 0u);
        if constexpr (NW == 1) v = make_uint4(~0u, ~0u, 0u, 0u);           // {key = EMPTY, count, pad}
        else if constexpr (NW == 2) { if ((i & 1) == 0) v = make_uint4(~0u, ~0u, ~0u, ~0u); }  // {w0, w1} = EMPTY
        else if (i % 3 != 2) v = make_uint4(~0u, ~0u, ~0u, ~0u);                               // {w0..w3} = EMPTY
        t[i] = v;
    }
}

// ------------------------------------------------------------------ export

// Bytes of one low.bin record for k.
KC_HD uint32_t kc_packed(uint32_t k) { return (k / 32) * 8 + (2 * (k % 32) + 7) / 8; }

// low.bin packing (src/ExportWriter.h:522-550): k/32 full words as raw
// little-endian u64, then the top ceil(2(k%32)/8) bytes of the tail word
// (masked to its 2(k%32) high bits), in little-endian byte order.
// One key packed at d (P bytes; full = k/32 whole words, tail_bytes of the
// masked tail word).
template <int NW>
KC_HD void pack_key(const typename KeyOf<NW>::T& key, uint8_t* d, uint32_t full,
                                         uint32_t tail_bytes, uint32_t P, uint64_t tmask) {
    // word f of the key (f < 4; words past the key's width read 0)
    auto word = [&](uint32_t f) -> uint64_t {
        if constexpr (NW == 1) {
            return f == 0 ? key : 0ull;
        } else if constexpr (NW == 2) {
            return f == 0 ? key.w0 : (f == 1 ? key.w1 : 0ull);
        } else {
            return f == 0 ? key.w0 : (f == 1 ? key.w1 : (f == 2 ? key.w2 : key.w3));
        }
    };
    if (P == 8) {
        *reinterpret_cast<uint64_t*>(d) = full ? word(0) : (word(0) & tmask);
    } else if (P == 16) {
        reinterpret_cast<uint64_t*>(d)[0] = word(0);
        reinterpret_cast<uint64_t*>(d)[1] = full == 2 ? word(1) : (word(1) & tmask);
    } else {
        // k/32 whole words little-endian, then the top tail_bytes bytes
        // of the masked tail word (src/ExportWriter.h:522-550): the record is
        // the little-endian byte string of the words w_0..w_{full-1}, t with
        // t = the masked tail word's top tail_bytes bytes.  d is a multiple
        // of P from an 8-byte aligned base, so it is aligned to P's lowest
        // set bit: stores of that width (1, 2 or 4 bytes) never straddle a
        // word of the string.
        const uint64_t t = tail_bytes ? (((full < 4 ? word(full) : 0ull) & tmask) >> (8 * (8 - tail_bytes))) : 0ull;
        auto sw = [&](uint32_t f) -> uint64_t { return f < full ? word(f) : t; };
        const uint32_t W = P & (0u - P);
        if (W >= 4) {
            for (uint32_t q = 0; q < P; q += 4)
                *reinterpret_cast<uint32_t*>(d + q) = (uint32_t)(sw(q >> 3) >> (8 * (q & 7)));
        } else if (W == 2) {
            for (uint32_t q = 0; q < P; q += 2)
                *reinterpret_cast<uint16_t*>(d + q) = (uint16_t)(sw(q >> 3) >> (8 * (q & 7)));
        } else {
            for (uint32_t q = 0; q < P; ++q) d[q] = (uint8_t)(sw(q >> 3) >> (8 * (q & 7)));
        }
    }
}

// Records of a run that a warp packs: the first occurrences of 32 segments
// from segment g on, lane l's segment holding n_l of them (0: left out),
// consecutive from dst (byte address, P bytes a record).  Every lane takes
// one record a round, whatever segment it lies in.  Records of whole words
// are stored as they are; others are assembled in the warp's buffer, which
// keeps dst's offset mod 16, and leave as 16-byte stores (bytes only at the
// run's two ends).  A store per record and 1..4 bytes kept the load/store
// unit busy instead: 1 M reads at k = 101 (88 M records of 26 bytes), count +
// histogram 18.6 -> 14.3 ms, of which the packing was 5.7.
constexpr int PACK_BUF = 16 + 32 * 32 + 16;
template <int NW>
__device__ __forceinline__ void pack_run(const typename KeyOf<NW>::T* __restrict__ keys, uint64_t g, uint32_t n_l,
                                         uint8_t* dst, uint32_t k, uint8_t* buf) {
    using K = typename KeyOf<NW>::T;
    constexpr int SEG = count_seg<NW>();
    const uint32_t full = k / 32, tail_bits = 2 * (k % 32), tail_bytes = (tail_bits + 7) / 8;
    const uint32_t P = full * 8 + tail_bytes;
    const uint64_t tmask = tail_bits ? (~0ull << (64 - tail_bits)) : 0ull;
    const uint32_t lane = threadIdx.x & 31;
    uint32_t incl = n_l;  // warp-inclusive running count
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
        if ((int)lane >= o) incl += y;
    }
    const uint32_t total = __shfl_sync(0xffffffffu, incl, 31);
    const uint32_t excl = incl - n_l;
    auto fetch = [&](uint32_t n, K& key) {  // record n of the run (any n: the shuffles are the warp's)
        uint32_t lo = 0, hi = 31;  // the first lane whose running count exceeds n
#pragma unroll
        for (int step = 0; step < 5; ++step) {
            const uint32_t mid = (lo + hi) >> 1;
            const uint32_t v = __shfl_sync(0xffffffffu, incl, mid);
            if (v > n) hi = mid;
            else lo = mid + 1;
        }
        const uint32_t e = __shfl_sync(0xffffffffu, excl, lo & 31);
        if (n < total) key = keys[(g + lo) * (uint64_t)SEG + (n - e)];
    };
    K key, next;
    fetch(lane, key);
    if (P % 8 == 0) {
        for (uint32_t n0 = 0; n0 < total; n0 += 32) {
            if (n0 + 32 < total) fetch(n0 + 32 + lane, next);
            if (n0 + lane < total) pack_key<NW>(key, dst + (uint64_t)(n0 + lane) * P, full, tail_bytes, P, tmask);
            key = next;
        }
        return;
    }
    const uint32_t head = (uint32_t)(reinterpret_cast<uintptr_t>(dst) & 15);
    uint8_t* out = dst - head;     // the buffer's byte 0
    uint32_t fill = head, skip = head;  // bytes in the buffer, of which the first `skip` are not this run's
    for (uint32_t n0 = 0; n0 < total; n0 += 32) {
        if (n0 + 32 < total) fetch(n0 + 32 + lane, next);
        const uint32_t m = min(32u, total - n0);
        if (lane < m) pack_key<NW>(key, buf + fill + lane * P, full, tail_bytes, P, tmask);
        __syncwarp();
        fill += m * P;
        const uint32_t vecs = fill >> 4;
        for (uint32_t v = lane; v < vecs; v += 32)
            if (v || !skip) reinterpret_cast<uint4*>(out)[v] = reinterpret_cast<const uint4*>(buf)[v];
        if (vecs) {
            if (skip && lane >= skip && lane < 16) out[lane] = buf[lane];
            skip = 0;
            uint4 rest = make_uint4(0u, 0u, 0u, 0u);
            if (lane == 0) rest = reinterpret_cast<const uint4*>(buf)[vecs];
            __syncwarp();
            if (lane == 0) *reinterpret_cast<uint4*>(buf) = rest;
            out += 16 * vecs;
            fill &= 15;
        }
        __syncwarp();
        key = next;
    }
    if (lane >= skip && lane < fill) out[lane] = buf[lane];  // fill < 16 here
    __syncwarp();  // the buffer is the next run's
}

// A warp packs 32 segments at a time: lane l loads segment l's count and
// output index (one coalesced load each).  WHOLE (records of whole words): the
// warp walks the segments that have first occurrences, B at a time, every
// lane loading all of its keys of those segments before storing any, so that
// 4 loads per lane are in flight; other records: pack_run.
template <int NW, bool WHOLE>
__global__ void pack_low(const void* routed, const uint32_t* seg_low, const uint64_t* seg_low_prefix, uint64_t n_segs,
                         uint32_t k, uint8_t* out, uint64_t out_base) {
    using K = typename KeyOf<NW>::T;
    constexpr int SEG = count_seg<NW>();
    constexpr int PER = SEG / 32;                  // keys per lane per segment
    constexpr int B = PER >= 4 ? 1 : 4 / PER;      // segments per round: 4 keys per lane in flight
    __shared__ __align__(16) uint8_t pack_buf[WHOLE ? 1 : 8][PACK_BUF];  // the launch has at most 8 warps
    const K* __restrict__ keys = reinterpret_cast<const K*>(routed);
    const uint32_t full = k / 32, tail_bits = 2 * (k % 32), tail_bytes = (tail_bits + 7) / 8;
    const uint32_t P = full * 8 + tail_bytes;
    const uint64_t tmask = tail_bits ? (~0ull << (64 - tail_bits)) : 0ull;
    const int lane = threadIdx.x & 31;
    const uint64_t warps = (uint64_t)gridDim.x * (blockDim.x >> 5);
    for (uint64_t g = ((uint64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * 32; g < n_segs;
         g += warps * 32) {
        const uint64_t my = g + lane;
        const uint32_t n_l = my < n_segs ? seg_low[my] : 0u;
        const uint64_t o_l = my < n_segs ? seg_low_prefix[my] : 0ull;
        if constexpr (!WHOLE) {
            const uint64_t o = __shfl_sync(0xffffffffu, o_l, 0);
            pack_run<NW>(keys, g, n_l, out + (out_base + o) * P, k, pack_buf[threadIdx.x >> 5]);
            continue;
        }
        uint32_t todo = WHOLE ? __ballot_sync(0xffffffffu, n_l != 0) : 0u;
        while (todo) {
            // B segments per round (warp-uniform picks from `todo`)
            uint32_t n[B];
            uint64_t o[B], s0[B];
#pragma unroll
            for (int b = 0; b < B; ++b) {
                const int q = todo ? __ffs(todo) - 1 : -1;
                todo &= todo - 1;
                const int src = q >= 0 ? q : 0;
                const uint32_t nq = __shfl_sync(0xffffffffu, n_l, src);
                const uint64_t oq = __shfl_sync(0xffffffffu, o_l, src);
                n[b] = q >= 0 ? nq : 0u;
                o[b] = out_base + oq;
                s0[b] = (g + (uint64_t)src) * (uint64_t)SEG;
            }
            K v[B][PER];
#pragma unroll
            for (int b = 0; b < B; ++b)
#pragma unroll
                for (int j = 0; j < PER; ++j) {
                    const uint32_t i = j * 32 + lane;
                    if (i < n[b]) v[b][j] = keys[s0[b] + i];
                }
#pragma unroll
            for (int b = 0; b < B; ++b)
#pragma unroll
                for (int j = 0; j < PER; ++j) {
                    const uint32_t i = j * 32 + lane;
                    if (i < n[b]) pack_key<NW>(v[b][j], out + (o[b] + i) * P, full, tail_bytes, P, tmask);
                }
        }
    }
}

// Work item of the table export: a range of one bucket's slots.
struct ExportChunk {
    uint64_t slot_begin;  // absolute slot index in the table arena
    uint32_t n_slots;
    uint32_t root;        // root file id of the bucket
};

template <int NW>
__device__ __forceinline__ bool slot_used(const typename SlotOf<NW>::T& s) {
    if constexpr (NW == 1) return s.key != EMPTY;
    else if constexpr (NW == 2) return !(s.w0 == EMPTY && s.w1 == EMPTY);
    else return s.state == SLOT_READY;
}

constexpr int EXP_THREADS = 256;
constexpr int EXP_ITEMS = 4;  // slots per thread per round (strided by EXP_THREADS)

// One ExportRecord<N> {key words, count, pad = 0} at index r.
template <int NW>
__device__ __forceinline__ void write_record(uint8_t* records, uint64_t r, const typename SlotOf<NW>::T& v) {
    if constexpr (NW == 1) {
        uint4 w;
        w.x = (uint32_t)v.key;
        w.y = (uint32_t)(v.key >> 32);
        w.z = v.count;
        w.w = 0;
        reinterpret_cast<uint4*>(records)[r] = w;
    } else if constexpr (NW == 2) {
        uint64_t* d = reinterpret_cast<uint64_t*>(records + r * 24);
        d[0] = v.w0;
        d[1] = v.w1;
        d[2] = (uint64_t)v.count;
    } else {
        uint64_t* d = reinterpret_cast<uint64_t*>(records + r * 40);
        d[0] = v.w0;
        d[1] = v.w1;
        d[2] = v.w2;
        d[3] = v.w3;
        d[4] = (uint64_t)v.count;
    }
}

// Count slots passing the filter min <= count <= max per export chunk and per
// root id (src/NewKmerTree.h:1159-1168), and occupied slots overall.  The
// per-chunk counts, scanned in chunk order, are the chunks' output offsets:
// chunks are listed root by root, so each root's records are contiguous.
// With `pass_bits` (chunks start at and span multiples of 32 slots), bit i of
// word w is set when arena slot 32w + i passes: a warp reads 32 consecutive
// slots, so one ballot is one word, and export_write_bits then reads only the
// passing slots.
template <int NW>
__global__ void __launch_bounds__(EXP_THREADS) export_count(const void* table, const ExportChunk* chunks,
                                                            uint64_t n_chunks, uint32_t min_c, uint32_t max_c,
                                                            uint32_t* chunk_pass, unsigned long long* root_count,
                                                            unsigned long long* occupied, uint32_t* pass_bits) {
    using S = typename SlotOf<NW>::T;
    __shared__ uint32_t s_pass[EXP_THREADS / 32], s_occ[EXP_THREADS / 32];
    const S* tab = reinterpret_cast<const S*>(table);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (uint64_t c = blockIdx.x; c < n_chunks; c += gridDim.x) {
        const ExportChunk ch = chunks[c];
        uint32_t pass = 0, occ = 0;
        for (uint32_t i0 = 0; i0 < ch.n_slots; i0 += EXP_THREADS * EXP_ITEMS) {
            S v[EXP_ITEMS];
#pragma unroll
            for (int j = 0; j < EXP_ITEMS; ++j) {
                const uint32_t i = i0 + j * EXP_THREADS + threadIdx.x;
                if (i < ch.n_slots) v[j] = tab[ch.slot_begin + i];
            }
#pragma unroll
            for (int j = 0; j < EXP_ITEMS; ++j) {
                const uint32_t i = i0 + j * EXP_THREADS + threadIdx.x;
                bool ok = false;
                if (i < ch.n_slots && slot_used<NW>(v[j])) {
                    ++occ;
                    ok = v[j].count >= min_c && v[j].count <= max_c;
                    pass += ok;
                }
                if (pass_bits) {
                    const uint32_t word = __ballot_sync(0xffffffffu, ok);
                    const uint32_t i_lane0 = i - (uint32_t)lane;
                    if (lane == 0 && i_lane0 < ch.n_slots) pass_bits[(ch.slot_begin + i_lane0) >> 5] = word;
                }
            }
        }
        for (int o = 16; o; o >>= 1) {
            pass += __shfl_xor_sync(0xffffffffu, pass, o);
            occ += __shfl_xor_sync(0xffffffffu, occ, o);
        }
        if (lane == 0) {
            s_pass[warp] = pass;
            s_occ[warp] = occ;
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            uint32_t tp = 0, to = 0;
            for (int w = 0; w < EXP_THREADS / 32; ++w) {
                tp += s_pass[w];
                to += s_occ[w];
            }
            chunk_pass[c] = tp;
            if (tp) atomicAdd(root_count + ch.root, (unsigned long long)tp);
            if (to) atomicAdd(occupied, (unsigned long long)to);
        }
        __syncthreads();
    }
}

// Write ExportRecord<N> {key words, count, pad = 0} of every passing slot,
// one read of the table: chunk c's records start at chunk_off[c] and follow
// table order (rounds of EXP_THREADS x EXP_ITEMS slots; inside a round, by
// thread, then item).  No atomics decide positions, so the record order is a
// function of the table alone.
template <int NW>
__global__ void __launch_bounds__(EXP_THREADS) export_write(const void* table, const ExportChunk* chunks,
                                                            uint64_t n_chunks, uint32_t min_c, uint32_t max_c,
                                                            const uint64_t* chunk_off, uint8_t* records) {
    using S = typename SlotOf<NW>::T;
    __shared__ uint32_t s_warp[EXP_THREADS / 32];
    const S* tab = reinterpret_cast<const S*>(table);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (uint64_t c = blockIdx.x; c < n_chunks; c += gridDim.x) {
        const ExportChunk ch = chunks[c];
        uint64_t out = chunk_off[c];
        for (uint32_t i0 = 0; i0 < ch.n_slots; i0 += EXP_THREADS * EXP_ITEMS) {
            S v[EXP_ITEMS];
            uint32_t keep = 0;
#pragma unroll
            for (int j = 0; j < EXP_ITEMS; ++j) {
                const uint32_t i = i0 + j * EXP_THREADS + threadIdx.x;
                if (i < ch.n_slots) {
                    v[j] = tab[ch.slot_begin + i];
                    if (slot_used<NW>(v[j]) && v[j].count >= min_c && v[j].count <= max_c) keep |= 1u << j;
                }
            }
            // block-wide exclusive scan of the per-thread keep counts
            const uint32_t mine = __popc(keep);
            uint32_t incl = mine;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += y;
            }
            if (lane == 31) s_warp[warp] = incl;
            __syncthreads();
            uint32_t before = 0, total = 0;
#pragma unroll
            for (int w = 0; w < EXP_THREADS / 32; ++w) {
                const uint32_t t = s_warp[w];
                before += w < warp ? t : 0u;
                total += t;
            }
            __syncthreads();  // s_warp is rewritten next round
            uint64_t r = out + before + incl - mine;
#pragma unroll
            for (int j = 0; j < EXP_ITEMS; ++j)
                if ((keep >> j) & 1u) write_record<NW>(records, r++, v[j]);
            out += total;
        }
    }
}

// export_write over the passing-slot bitmap of export_count.  Per round a
// warp covers 32 bitmap words (1024 slots) and lane l of each pass takes the
// warp's l-th passing slot: the owning word by a binary search over the
// lanes' running popcounts, the bit by nth_set_bit.  Every lane reads one slot per
// pass and consecutive lanes write consecutive records, in table order (the
// order export_write produces).
template <int NW>
__global__ void __launch_bounds__(EXP_THREADS) export_write_bits(const void* table, const uint32_t* pass_bits,
                                                                 const ExportChunk* chunks, uint64_t n_chunks,
                                                                 const uint64_t* chunk_off, uint8_t* records) {
    using S = typename SlotOf<NW>::T;
    __shared__ uint32_t s_warp[EXP_THREADS / 32];
    const S* tab = reinterpret_cast<const S*>(table);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (uint64_t c = blockIdx.x; c < n_chunks; c += gridDim.x) {
        const ExportChunk ch = chunks[c];
        const uint64_t w0 = ch.slot_begin >> 5;
        const uint32_t nw = ch.n_slots >> 5;
        uint64_t out = chunk_off[c];
        for (uint32_t r0 = 0; r0 < nw; r0 += EXP_THREADS) {
            const uint32_t wi = r0 + threadIdx.x;
            const uint32_t m = wi < nw ? __ldcg(pass_bits + w0 + wi) : 0u;
            uint32_t incl = __popc(m);  // warp-inclusive running count
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += y;
            }
            const uint32_t wtot = __shfl_sync(0xffffffffu, incl, 31);
            if (lane == 31) s_warp[warp] = wtot;
            __syncthreads();
            uint32_t before = 0, total = 0;
#pragma unroll
            for (int w = 0; w < EXP_THREADS / 32; ++w) {
                const uint32_t t = s_warp[w];
                before += w < warp ? t : 0u;
                total += t;
            }
            __syncthreads();  // s_warp is rewritten next round
            const uint64_t base = out + before;
            const uint64_t cell_w = (w0 + r0 + (uint32_t)warp * 32) << 5;  // first slot of lane 0's word
            for (uint32_t n0 = 0; n0 < wtot; n0 += 32) {
                const uint32_t n = n0 + lane;
                // owner lane q: the first lane whose running count exceeds n
                uint32_t lo = 0, hi = 31;
#pragma unroll
                for (int step = 0; step < 5; ++step) {
                    const uint32_t mid = (lo + hi) >> 1;
                    const uint32_t v = __shfl_sync(0xffffffffu, incl, mid);
                    if (v > n) hi = mid;
                    else lo = mid + 1;
                }
                const uint32_t q = lo;
                const uint32_t mq = __shfl_sync(0xffffffffu, m, q);
                const uint32_t eq = __shfl_sync(0xffffffffu, incl, q) - __popc(mq);  // passing slots before word q
                if (n < wtot) {
                    const uint32_t bit = nth_set_bit(mq, n - eq);
                    const S v = tab[cell_w + ((uint64_t)q << 5) + bit];
                    write_record<NW>(records, base + n, v);
                }
            }
            out += total;
        }
    }
}

// ------------------------------------------------------ merged histogram
//
// Device form of tool/histogram_tool.cpp "precise"
// (tool/HighFrequencyInsertThreadPool.h:150-177,
// tool/LowFrequencyQueryThreadPool.h:375-432): exact count of a key = its
// table count + [key in low.bin].  A key is in low.bin at most once, so the
// histogram is a sum in any order: +1 at its count for every table key; for
// every low.bin key +1 at count 1 when no table holds it, else -1 at its
// table count and +1 at the next.  Nothing is written to the tables.  Keys in
// low.bin order visit a bucket's table at random, so a low.bin key is looked
// up where its table slice is at hand: in shared memory, window by window,
// after a windowed count (hist_window in kc_window.cuh), else in L2.
// Histogram bins are aggregated per CTA in shared memory (HIST_SMEM bins;
// larger counts go straight to global atomics).

constexpr int HIST_SMEM = 512;

// Key of low.bin record r (layout of src/ExportWriter.h:522-550, read back as
// tool/ExportReader.h:355-391 does).  Records of a multiple of 8 bytes
// (k = 29..32, 61..64, 93..96, 125..128) are read as aligned words.
template <int NW>
__device__ __forceinline__ typename KeyOf<NW>::T unpack_low(const uint8_t* low, uint64_t r, uint32_t P, uint32_t full,
                                                            uint32_t tail_bytes) {
    const uint8_t* p = low + r * P;
    uint64_t w[4] = {0, 0, 0, 0};
    if ((P & 7u) == 0) {
        const uint64_t* q = reinterpret_cast<const uint64_t*>(p);
        for (uint32_t f = 0; f < P / 8 && f < (uint32_t)NW; ++f) w[f] = q[f];
    } else {
        for (uint32_t f = 0; f < full; ++f)
            for (uint32_t b = 0; b < 8; ++b) w[f] |= (uint64_t)p[8 * f + b] << (8 * b);
        for (uint32_t b = 0; b < tail_bytes; ++b) w[full] |= (uint64_t)p[8 * full + b] << (8 * (8 - tail_bytes + b));
    }
    typename KeyOf<NW>::T key;
    if constexpr (NW == 1) key = w[0];
    else if constexpr (NW == 2) key = Key2{w[0], w[1]};
    else key = Key4{w[0], w[1], w[2], w[3]};
    return key;
}

// The same with at most NW + 1 aligned word loads for any record size: the
// buffer must be readable for 8 (NW + 1) bytes from the word a record starts
// in (the context's packed low.bin buffer keeps 64 bytes after its last one).
template <int NW>
__device__ __forceinline__ typename KeyOf<NW>::T load_low(const uint8_t* __restrict__ low, uint64_t r, uint32_t P,
                                                          uint32_t full, uint32_t tail_bytes) {
    uint64_t w[NW];
    const uint64_t a = r * P;
    const uint64_t* q = reinterpret_cast<const uint64_t*>(low) + (a >> 3);
    const uint32_t sh = (uint32_t)(a & 7) * 8;
    if (P == 8 * NW) {
#pragma unroll
        for (int i = 0; i < NW; ++i) w[i] = __ldcs(q + i);
    } else {
        uint64_t x[NW + 1];
#pragma unroll
        for (int i = 0; i <= NW; ++i) x[i] = __ldg(q + i);
#pragma unroll
        for (int i = 0; i < NW; ++i) {
            const uint64_t v = sh ? (x[i] >> sh) | (x[i + 1] << (64 - sh)) : x[i];
            w[i] = (uint32_t)i < full ? v : ((uint32_t)i == full && tail_bytes ? v << (64 - 8 * tail_bytes) : 0ull);
        }
    }
    if constexpr (NW == 1) return w[0];
    else if constexpr (NW == 2) return Key2{w[0], w[1]};
    else return Key4{w[0], w[1], w[2], w[3]};
}

// Table lookups.  A key is stored at most PROBE_LIMIT - 1 cells after its
// first one, with no EMPTY cell in between.
template <int NW>
struct Cell {  // what one probe reads
    typename KeyOf<NW>::T key;
    uint32_t count;  // 256-bit cells: read only when the key matches
    bool used;
};
template <int NW>
__device__ __forceinline__ Cell<NW> read_cell_all(const typename SlotOf<NW>::T* s) {
    Cell<NW> c;
    if constexpr (NW == 1) {
        const uint4 v = __ldcg(reinterpret_cast<const uint4*>(s));
        c.key = ((uint64_t)v.y << 32) | v.x;
        c.count = v.z;
        c.used = c.key != EMPTY;
    } else if constexpr (NW == 2) {
        const ulonglong2 v = __ldcg(reinterpret_cast<const ulonglong2*>(s));
        c.key = Key2{v.x, v.y};
        c.count = 0;
        c.used = !(v.x == EMPTY && v.y == EMPTY);
    } else {
        const ulonglong2 a = __ldcg(reinterpret_cast<const ulonglong2*>(s));
        const ulonglong2 b = __ldcg(reinterpret_cast<const ulonglong2*>(s) + 1);
        const uint2 t = __ldcg(reinterpret_cast<const uint2*>(s) + 4);
        c.key = Key4{a.x, a.y, b.x, b.y};
        c.count = t.x;
        c.used = t.y == SLOT_READY;  // after the count every used slot is ready
    }
    return c;
}

// `add` keys of exact count `merged` (add may be -1: bins and totals are
// two's complement sums).
__device__ __forceinline__ void hist_add(uint32_t* sh, unsigned long long* gh, uint64_t merged, int add, uint32_t lo,
                                         uint32_t hi) {
    if (merged < lo || merged > hi) return;
    const uint64_t bin = merged - lo;
    if (bin < HIST_SMEM) atomicAdd(sh + bin, (uint32_t)add);
    else atomicAdd(gh + bin, (unsigned long long)(long long)add);
}
__device__ __forceinline__ void hist_flush(const uint32_t* sh, unsigned long long* gh, uint32_t lo, uint32_t hi) {
    for (int i = threadIdx.x; i < HIST_SMEM; i += blockDim.x)
        if (sh[i] && (uint64_t)lo + i <= hi) atomicAdd(gh + i, (unsigned long long)(long long)(int)sh[i]);
}

// Table placement of a bucket in 16 bytes.
struct TabRef {
    uint64_t off, mask;
};
// The buckets' table placements in shared memory when there are at most 256
// of them (a lookup per key through L1 otherwise).
struct TabRefs {
    const BucketMeta* meta;
    const TabRef* sm;
    __device__ __forceinline__ TabRef operator()(uint32_t b) const {
        return sm ? sm[b] : TabRef{__ldg(&meta[b].tab_off), __ldg(&meta[b].tab_mask)};
    }
};
constexpr uint32_t TABREF_SMEM = 256;
__device__ __forceinline__ TabRefs tab_refs(const BucketMeta* meta, uint32_t n_buckets, TabRef* sm) {
    if (n_buckets > TABREF_SMEM) return TabRefs{meta, nullptr};
    for (uint32_t b = threadIdx.x; b < n_buckets; b += blockDim.x) sm[b] = TabRef{meta[b].tab_off, meta[b].tab_mask};
    return TabRefs{meta, sm};  // the caller's __syncthreads publishes sm
}

// Items a lane of the lookup kernels resolves side by side: the next record
// and the first cell of each are in flight together.
template <int NW>
constexpr int lookup_items() {
    return NW == 4 ? 1 : 2;
}

// Calls found(key, count) for every low.bin record [r0, r1) that its bucket's
// table holds and returns how many this thread found.  A warp probes in
// lockstep rounds (the vote ends a round for all its lanes): left to itself
// the compiler lets lanes that leave the probe loop early run the rest of it
// apart, which cost 940 warp instructions per 32 keys of 128 bits where the
// rounds take about 200.
template <int NW, class F>
__device__ __forceinline__ uint32_t lookup_low(const uint8_t* __restrict__ low, uint64_t r0, uint64_t r1, uint32_t k,
                                               uint32_t bucket_shift, const TabRefs& refs,
                                               const typename SlotOf<NW>::T* __restrict__ table, F found) {
    using K = typename KeyOf<NW>::T;
    using S = typename SlotOf<NW>::T;
    constexpr int IT = lookup_items<NW>();
    const uint32_t full = k / 32, tail_bytes = (2 * (k % 32) + 7) / 8, P = full * 8 + tail_bytes;
    const uint64_t step = (uint64_t)gridDim.x * blockDim.x;
    const uint32_t lane = threadIdx.x & 31;
    uint32_t n = 0;
    // r: the warp's first record of the round
    for (uint64_t r = r0 + (uint64_t)blockIdx.x * blockDim.x + (threadIdx.x & ~31u); r < r1; r += step * IT) {
        K key[IT];
        const S* tab[IT];
        uint32_t at[IT], mask[IT];
        Cell<NW> c[IT];
        uint32_t todo = 0, hit = 0;
#pragma unroll
        for (int j = 0; j < IT; ++j) {
            const uint64_t i = r + j * step + lane;
            if (i < r1) {
                key[j] = load_low<NW>(low, i, P, full, tail_bytes);
                todo |= 1u << j;
            }
        }
#pragma unroll
        for (int j = 0; j < IT; ++j)
            if ((todo >> j) & 1u) {
                const TabRef t = refs((uint32_t)(key_hi(key[j]) >> bucket_shift));
                tab[j] = table + t.off;
                mask[j] = (uint32_t)t.mask;  // a bucket holds fewer than 2^32 cells
                at[j] = (uint32_t)(hash_key(key[j]) >> 17) & mask[j];
                c[j] = read_cell_all<NW>(tab[j] + at[j]);
            }
        for (uint32_t p = 0;; ++p) {
#pragma unroll
            for (int j = 0; j < IT; ++j) {
                if (!((todo >> j) & 1u)) continue;
                const bool eq = c[j].used && same_key(c[j].key, key[j]);
                if (eq) hit |= 1u << j;
                if (eq || !c[j].used || p >= min((uint32_t)PROBE_LIMIT - 1, mask[j])) todo &= ~(1u << j);
            }
            if (!__any_sync(0xffffffffu, todo != 0)) break;  // warp-uniform
#pragma unroll
            for (int j = 0; j < IT; ++j)
                if ((todo >> j) & 1u) {
                    at[j] = (at[j] + 1) & mask[j];
                    c[j] = read_cell_all<NW>(tab[j] + at[j]);
                }
        }
#pragma unroll
        for (int j = 0; j < IT; ++j)
            if ((hit >> j) & 1u) {
                if constexpr (NW == 2) c[j].count = __ldcg(&tab[j][at[j]].count);
                found(key[j], c[j].count);
                ++n;
            }
        __syncwarp();
    }
    return n;
}

// Sum of v over the block, added to *out by one thread.
__device__ __forceinline__ void block_add(unsigned long long* out, long long v, unsigned long long* s_sum) {
    for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if ((threadIdx.x & 31) == 0 && v) atomicAdd(s_sum, (unsigned long long)v);
    __syncthreads();
    if (threadIdx.x == 0 && *s_sum) atomicAdd(out, *s_sum);
}

// First low.bin record of output segment `seg` of a batch whose segments'
// record offsets are prefix[0..nsegs) and that holds n_low records.
__device__ __forceinline__ uint64_t low_at(const uint64_t* prefix, uint64_t nsegs, uint64_t seg, uint64_t n_low) {
    return seg < nsegs ? prefix[seg] : n_low;
}

// Low.bin records of the segments from first_seg on (0 without a prefix: all
// n_low records): histogram changes of those some table holds, +1 at count 1
// for the others.  extra -= the number found (distinct keys = low.bin keys +
// table keys - found).
template <int NW>
__global__ void __launch_bounds__(256, 5) hist_low_pass(const uint8_t* low, uint64_t n_low, const uint64_t* prefix,
                                                        uint64_t nsegs, uint64_t first_seg, uint32_t k,
                                                        const BucketMeta* meta, uint32_t n_buckets,
                                                        uint32_t bucket_shift, const void* table, uint32_t lo,
                                                        uint32_t hi, unsigned long long* gh,
                                                        unsigned long long* extra) {
    __shared__ uint32_t sh[HIST_SMEM];
    __shared__ TabRef s_ref[TABREF_SMEM];
    __shared__ unsigned long long s_found;
    for (int i = threadIdx.x; i < HIST_SMEM; i += blockDim.x) sh[i] = 0;
    if (threadIdx.x == 0) s_found = 0;
    const TabRefs refs = tab_refs(meta, n_buckets, s_ref);
    __syncthreads();
    const uint64_t r0 = prefix ? low_at(prefix, nsegs, first_seg, n_low) : 0;
    const uint32_t n = lookup_low<NW>(low, r0, n_low, k, bucket_shift, refs,
                                      reinterpret_cast<const typename SlotOf<NW>::T*>(table),
                                      [&](const typename KeyOf<NW>::T&, uint32_t count) {
                                          hist_add(sh, gh, count, -1, lo, hi);
                                          hist_add(sh, gh, (uint64_t)count + 1, 1, lo, hi);
                                      });
    block_add(extra, -(long long)n, &s_found);  // synchronises the block: sh is complete
    hist_flush(sh, gh, lo, hi);
    // the records no table holds: all minus those found, at count 1
    if (threadIdx.x == 0 && lo <= 1) {
        const long long all = blockIdx.x == 0 ? (long long)(n_low - r0) : 0;
        const long long add = all + (long long)s_found;  // s_found = -(found by this block)
        if (add) atomicAdd(gh + (1 - lo), (unsigned long long)add);
    }
}

// Every table key at its table count; extra += the number of table keys.
template <int NW>
__global__ void __launch_bounds__(256) hist_table_pass(const void* table, const ExportChunk* chunks, uint64_t n_chunks,
                                                       uint32_t lo, uint32_t hi, unsigned long long* gh,
                                                       unsigned long long* extra) {
    using S = typename SlotOf<NW>::T;
    __shared__ uint32_t sh[HIST_SMEM];
    __shared__ unsigned long long s_used;
    for (int i = threadIdx.x; i < HIST_SMEM; i += blockDim.x) sh[i] = 0;
    if (threadIdx.x == 0) s_used = 0;
    __syncthreads();
    uint32_t n = 0;
    for (uint64_t c = blockIdx.x; c < n_chunks; c += gridDim.x) {
        const ExportChunk ch = chunks[c];
        const S* t = reinterpret_cast<const S*>(table) + ch.slot_begin;
#pragma unroll 4
        for (uint32_t q = threadIdx.x; q < ch.n_slots; q += blockDim.x) {
            const S s = t[q];
            if (slot_used<NW>(s)) {
                ++n;
                hist_add(sh, gh, s.count, 1, lo, hi);
            }
        }
    }
    block_add(extra, (long long)n, &s_used);
    hist_flush(sh, gh, lo, hi);
}

// Per model bucket (key word 0 >> 52) loads of the last result, as the
// histogram's sums: distinct = low.bin keys + table keys - low.bin keys found
// in a table; kmers = low.bin keys + the table keys' counts.
// model buckets of the sizing loads (the top 12 bits of the key)
constexpr uint32_t KC_LOADS_BINS = 4096;
// dynamic shared memory of loads_low_pass / loads_table_pass
constexpr size_t loads_low_smem() { return KC_LOADS_BINS * (4 + 4); }
constexpr size_t loads_table_smem() { return KC_LOADS_BINS * (8 + 4); }

template <int NW>
__global__ void __launch_bounds__(512) loads_low_pass(const uint8_t* low, uint64_t n_low, uint32_t k,
                                                      const BucketMeta* meta, uint32_t n_buckets,
                                                      uint32_t bucket_shift, const void* table,
                                                      unsigned long long* distinct, unsigned long long* kmers) {
    // per-CTA totals per model bucket in shared memory (consecutive low keys
    // share their model bucket, so global atomics would serialise on it),
    // added to the global totals once per CTA
    extern __shared__ unsigned long long ld_smem[];
    uint32_t* s_low = reinterpret_cast<uint32_t*>(ld_smem);  // [KC_LOADS_BINS]
    uint32_t* s_found = s_low + KC_LOADS_BINS;               // [KC_LOADS_BINS]
    __shared__ TabRef s_ref[TABREF_SMEM];
    for (uint32_t i = threadIdx.x; i < 2 * KC_LOADS_BINS; i += blockDim.x) s_low[i] = 0;
    const TabRefs refs = tab_refs(meta, n_buckets, s_ref);
    __syncthreads();
    lookup_low<NW>(low, 0, n_low, k, bucket_shift, refs, reinterpret_cast<const typename SlotOf<NW>::T*>(table),
                   [&](const typename KeyOf<NW>::T& key, uint32_t) { atomicAdd(s_found + (key_hi(key) >> 52), 1u); });
    const uint32_t full = k / 32, tail_bytes = (2 * (k % 32) + 7) / 8, P = full * 8 + tail_bytes;
    for (uint64_t r = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; r < n_low; r += (uint64_t)gridDim.x * blockDim.x)
        atomicAdd(s_low + (key_hi(load_low<NW>(low, r, P, full, tail_bytes)) >> 52), 1u);
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < KC_LOADS_BINS; i += blockDim.x) {
        if (s_low[i] != s_found[i]) atomicAdd(distinct + i, (unsigned long long)s_low[i] - s_found[i]);
        if (s_low[i]) atomicAdd(kmers + i, (unsigned long long)s_low[i]);
    }
}

template <int NW>
__global__ void loads_table_pass(const void* table, const ExportChunk* chunks, uint64_t n_chunks,
                                 unsigned long long* distinct, unsigned long long* tkeys, unsigned long long* kmers) {
    extern __shared__ unsigned long long ld_smem[];
    unsigned long long* s_kmers = ld_smem;                                     // [KC_LOADS_BINS]
    uint32_t* s_tkeys = reinterpret_cast<uint32_t*>(ld_smem + KC_LOADS_BINS);  // [KC_LOADS_BINS]
    for (uint32_t i = threadIdx.x; i < KC_LOADS_BINS; i += blockDim.x) {
        s_kmers[i] = 0;
        s_tkeys[i] = 0;
    }
    __syncthreads();
    using S = typename SlotOf<NW>::T;
    for (uint64_t c = blockIdx.x; c < n_chunks; c += gridDim.x)
    for (uint32_t q = threadIdx.x; q < chunks[c].n_slots; q += blockDim.x) {
        const S s = reinterpret_cast<const S*>(table)[chunks[c].slot_begin + q];
        if (!slot_used<NW>(s)) continue;
        uint64_t hi;
        if constexpr (NW == 1) hi = s.key;
        else hi = s.w0;
        atomicAdd(s_tkeys + (hi >> 52), 1u);
        atomicAdd(s_kmers + (hi >> 52), (unsigned long long)s.count);
    }
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < KC_LOADS_BINS; i += blockDim.x) {
        if (s_tkeys[i]) {
            atomicAdd(tkeys + i, (unsigned long long)s_tkeys[i]);
            atomicAdd(distinct + i, (unsigned long long)s_tkeys[i]);
            atomicAdd(kmers + i, s_kmers[i]);
        }
    }
}

// EMPTY keys into the unfilled tail of each estimated bucket region:
// routed[min(cursor[b], region_fill[b], region_end[b]), region_end[b]).
template <int NW>
__global__ void fill_region_gaps(void* routed, const unsigned long long* cursor, const unsigned long long* region_fill,
                                 const unsigned long long* region_end, uint32_t n_buckets) {
    using K = typename KeyOf<NW>::T;
    K* keys = reinterpret_cast<K*>(routed);
    const uint32_t b = blockIdx.x;
    if (b >= n_buckets) return;
    const unsigned long long end = region_end[b];
    for (unsigned long long i = min(min(cursor[b], region_fill[b]), end) + threadIdx.x; i < end; i += blockDim.x) {
        if constexpr (NW == 1) keys[i] = EMPTY;
        else if constexpr (NW == 2) keys[i] = Key2{EMPTY, EMPTY};
        else keys[i] = Key4{EMPTY, EMPTY, EMPTY, EMPTY};
    }
}

// ------------------------------------------------------- multi-set batches

// EMPTY keys into the alignment gap after each set's routed region.
template <int NW>
__global__ void fill_set_gaps(void* routed, const uint64_t* set_end_key, const uint64_t* set_next_key, uint32_t n_sets) {
    using K = typename KeyOf<NW>::T;
    K* keys = reinterpret_cast<K*>(routed);
    const uint32_t s = blockIdx.x;
    if (s >= n_sets) return;
    for (uint64_t i = set_end_key[s] + threadIdx.x; i < set_next_key[s]; i += blockDim.x) {
        if constexpr (NW == 1) keys[i] = EMPTY;
        else if constexpr (NW == 2) keys[i] = Key2{EMPTY, EMPTY};
        else keys[i] = Key4{EMPTY, EMPTY, EMPTY, EMPTY};
    }
}

// Pack first occurrences of a multi-set batch: segment sg of set s writes at
// low_byte_base[s] (a multiple of 16) + (prefix[sg] - prefix[first segment
// of s]) * P(k_s).  A warp takes 32 segments at a time (each lane finds its
// segment's set and output place) and packs the segments of one set after
// those of another.
template <int NW>
__global__ void pack_low_sets(const void* routed, const uint32_t* seg_low, const uint64_t* seg_low_prefix, uint64_t n_segs,
                              const uint64_t* set_seg_start, const uint32_t* set_k, const uint64_t* low_byte_base,
                              uint32_t n_sets, uint8_t* out) {
    using K = typename KeyOf<NW>::T;
    __shared__ __align__(16) uint8_t pack_buf[8][PACK_BUF];  // the launch has at most 8 warps
    const K* __restrict__ keys = reinterpret_cast<const K*>(routed);
    const int lane = threadIdx.x & 31;
    const uint64_t warps = (uint64_t)gridDim.x * (blockDim.x >> 5);
    for (uint64_t g = ((uint64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * 32; g < n_segs;
         g += warps * 32) {
        const uint64_t my = g + lane;
        uint32_t n_l = 0, set = 0;
        uint64_t dst_l = 0;
        if (my < n_segs && (n_l = seg_low[my]) != 0) {
            uint32_t lo = 0, hi = n_sets;
            while (hi - lo > 1) {
                const uint32_t mid = (lo + hi) / 2;
                if (set_seg_start[mid] <= my) lo = mid;
                else hi = mid;
            }
            set = lo;
            dst_l = low_byte_base[lo] + (seg_low_prefix[my] - seg_low_prefix[set_seg_start[lo]]) * kc_packed(set_k[lo]);
        }
        uint32_t todo = __ballot_sync(0xffffffffu, n_l != 0);
        while (todo) {
            const int q = __ffs(todo) - 1;
            const uint32_t qset = __shfl_sync(0xffffffffu, set, q);
            const uint64_t dst = __shfl_sync(0xffffffffu, dst_l, q);
            const uint32_t run = __ballot_sync(0xffffffffu, n_l != 0 && set == qset);
            todo &= ~run;
            pack_run<NW>(keys, g, ((run >> lane) & 1u) ? n_l : 0u, out + dst, set_k[qset], pack_buf[threadIdx.x >> 5]);
        }
    }
}

}  // namespace kc
