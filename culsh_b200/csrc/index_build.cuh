// Bucket boundaries and offsets from the sorted (key, row) pairs.  Replaces
// mark_boundaries_kernel + ExclusiveSum + Select::Flagged + build_final_index_kernel
// (core/fit.cuh:97-208, 285-363).  The sorted keys sit next to each other, so a boundary
// is a compare of two adjacent keys (no gather of signatures through the permutation),
// the sorted row ids already are all_candidate_indices, and one count pass + one write
// pass produce bucket keys, bucket offsets and table offsets; a self-join takes the list of every
// (table, row) from the finished buckets (bucket_bounds_kernel).
#pragma once

#include "common.cuh"
#include "radix_sort.cuh"

namespace culsh_b200 {

constexpr int IB_THREADS = 256;
constexpr int IB_IPT = 8;
constexpr int IB_TILE = IB_THREADS * IB_IPT;
constexpr int IB_WORDS = IB_TILE / 32;  // head bits of a tile

template <int NW>
__device__ __forceinline__ bool keys_differ(const uint32_t* __restrict__ a,
                                            const uint32_t* __restrict__ b) {
    bool d = false;
#pragma unroll
    for (int w = 0; w < NW; ++w) d |= a[w] != b[w];
    return d;
}

// heads per tile, and a bit per item that is one: heads[tile][IB_WORDS].  A tile covers IB_TILE consecutive items of one table
template <int NW>
__global__ void __launch_bounds__(IB_THREADS)
bucket_count_kernel(const uint32_t* __restrict__ keys, int n, int tiles_per_table,
                    uint32_t* __restrict__ tile_heads, uint32_t* __restrict__ heads, KernelBefore kernel_before) {
    behind_kernel_before(keys, tile_heads, heads, kernel_before);
    __shared__ uint32_t s_warp[32];
    const int t = blockIdx.x / tiles_per_table;
    const int lt = blockIdx.x - t * tiles_per_table;
    const size_t tbase = (size_t)t * n;
    // a warp takes IB_IPT * 32 items next to one another, and lane i keeps word i of their bits
    const int lane = threadIdx.x & 31, first = (threadIdx.x >> 5) * (IB_IPT * 32);
    uint32_t mine = 0;
#pragma unroll
    for (int i = 0; i < IB_IPT; ++i) {
        const int li = lt * IB_TILE + first + i * 32 + lane;
        bool head = false;
        if (li < n) head = li == 0 || keys_differ<NW>(keys + (tbase + li) * NW, keys + (tbase + li - 1) * NW);
        const uint32_t word = __ballot_sync(0xFFFFFFFFu, head);
        if (lane == i) mine = word;
    }
    if (lane < IB_IPT) heads[(size_t)blockIdx.x * IB_WORDS + (first >> 5) + lane] = mine;
    uint32_t total;
    block_exclusive_scan<uint32_t>((uint32_t)__popc(mine), s_warp, total);
    if (threadIdx.x == 0) tile_heads[blockIdx.x] = total;
}

// tile_base: exclusive scan of tile_heads (tile_base[n_tiles] = B).
// A prefix over the words of head bits gives every head its bucket id; keys are read only where there is one, and bucket
// keys / offsets go to consecutive addresses.  (With the keys read and compared once more instead of the bits: 12.5M x 16 keys of two words 660 -> 469 us, with the count 967 -> 779; 10M x 48 of one 925 -> 582, with the count 1,425 -> 1,143.)
template <int NW>
__global__ void __launch_bounds__(IB_THREADS)
bucket_write_kernel(const uint32_t* __restrict__ keys, int n, int L, int tiles_per_table,
                    const uint32_t* __restrict__ tile_base, uint32_t n_tiles, const uint32_t* __restrict__ heads,
                    uint32_t* __restrict__ bucket_keys, int32_t* __restrict__ bucket_offsets,
                    int32_t* __restrict__ table_offsets, KernelBefore kernel_before) {
    behind_kernel_before(keys, tile_base, heads, bucket_keys, bucket_offsets, table_offsets, kernel_before);
    constexpr int WORDS = IB_WORDS;
    __shared__ uint32_t s_bits[WORDS];
    __shared__ uint32_t s_pref[WORDS];
    const int t = blockIdx.x / tiles_per_table;
    const int lt = blockIdx.x - t * tiles_per_table;
    const size_t tbase = (size_t)t * n;
    const int lane = threadIdx.x & 31;
    const uint32_t base_bucket = tile_base[blockIdx.x];
    if (threadIdx.x < WORDS) s_bits[threadIdx.x] = heads[(size_t)blockIdx.x * WORDS + threadIdx.x];
    __syncthreads();
    if (threadIdx.x < 32) {  // exclusive prefix of the pop-counts of the WORDS ballot words
        uint32_t run = 0;
        for (int w0 = 0; w0 < WORDS; w0 += 32) {
            const uint32_t c = __popc(s_bits[w0 + lane]);
            uint32_t inc = c;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                uint32_t x = __shfl_up_sync(0xFFFFFFFFu, inc, o);
                if (lane >= o) inc += x;
            }
            s_pref[w0 + lane] = run + inc - c;
            run += __shfl_sync(0xFFFFFFFFu, inc, 31);
        }
    }
    __syncthreads();
    if (lt == 0 && threadIdx.x == 0) table_offsets[t] = (int32_t)base_bucket;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        uint32_t B = tile_base[n_tiles];
        table_offsets[L] = (int32_t)B;
        bucket_offsets[B] = (int32_t)((size_t)n * L);
    }
#pragma unroll
    for (int i = 0; i < IB_IPT; ++i) {
        const int local = i * IB_THREADS + threadIdx.x;
        const int li = lt * IB_TILE + local;
        if (li >= n) continue;
        const uint32_t word = s_bits[local >> 5];
        const bool head = (word >> lane) & 1u;
        // heads up to and including this item, minus one = bucket of the item
        const uint32_t bid = base_bucket + s_pref[local >> 5] + __popc(word & (0xFFFFFFFFu >> (31 - lane))) - 1u;
        if (head) {
            if (bucket_keys) {  // null in a self-join, which looks nothing up
                const uint32_t* kp = keys + (tbase + li) * NW;
                uint32_t kk[NW];
                load_key<NW>(kp, kk);
                store_key<NW>(bucket_keys + (size_t)bid * NW, kk);
            }
            bucket_offsets[bid] = (int32_t)(tbase + li);
        }
    }
}

// sort_ctas: CTAs for each table that sorted in the one launch in front, if there was one.  They leave their SMs one by one, and this kernel's CTAs, a
// few for each SM, gather on the first where they are launched early.  With long keys and many tables that costs more than it saves.  Whole fits before early
// launches, with all of them, and as it is: 148 tables of 3,000 keys of 64 bytes 400, 499 and 396 us, 32 of 8,192 486, 581 and 480, 48 of 5,000
// 415, 435 and 414, 148 of 3,000 keys of 12 bytes 119, 120 and 115.
template <int NW>
inline void launch_bucket_count(const CtxPtr& c, const uint32_t* keys, int n, int L, int sort_ctas,
                                uint32_t* tile_heads, uint32_t* heads) {
    int tpt = (int)ceil_div(n, IB_TILE);
    const bool early = NW < 4 || (size_t)std::max(sort_ctas, 0) * L * NW < 2 * (size_t)c->sm_count;
    launch_with(early, c->stream, bucket_count_kernel<NW>, (size_t)tpt * L, 1u, IB_THREADS, 0, keys, n, tpt, tile_heads, heads);
    KERNEL_CHECK();
}

template <int NW>
inline void launch_bucket_write(cudaStream_t s, const uint32_t* keys, int n, int L, const uint32_t* tile_base, const uint32_t* heads,
                                uint32_t* bucket_keys, int32_t* bucket_offsets, int32_t* table_offsets) {
    int tpt = (int)ceil_div(n, IB_TILE);
    uint32_t n_tiles = (uint32_t)((size_t)tpt * L);
    launch_next(s, bucket_write_kernel<NW>, n_tiles, IB_THREADS, 0, keys, n, L, tpt, tile_base, n_tiles, heads, bucket_keys,
                                                          bucket_offsets, table_offsets);
    KERNEL_CHECK();
}

// Self-join: the list of every (table, row), packed into one word, packed[t * n + row]:
//   0                          the row is alone in its bucket
//   PB_PAIR | other row        the bucket has two rows (only if asked for)
//   position | rows << pos_bits  position of the list inside the table; the largest number of rows
//                              stands for "that many or more", and the reader looks the end up
// Half of the lists that are worth a look hold two rows: with the other one at hand the gather
// leaves the random read of the list out.
constexpr uint32_t PB_PAIR = 0x80000000u;
struct PackedBounds {
    int pos_bits;       // bits of n - 1, at most 30
    uint32_t max_len;   // 2^(31 - pos_bits) - 1
};
inline PackedBounds packed_bounds(int n) {
    int bits = 1;
    while (bits < 29 && ((uint32_t)(n - 1) >> bits)) ++bits;
    if ((uint32_t)(n - 1) >> bits) ++bits;
    return PackedBounds{bits, 0x7FFFFFFFu >> bits};
}

// `packed` comes zeroed and buckets of one row are left out: they add nothing but the row itself,
// which the gather supplies, and they are the larger part (10M x 48 tables: 250M of 480M items).
// A CTA takes the same IB_TILE consecutive items as bucket_write_kernel: the offsets of the buckets
// that meet the tile come in one coalesced read, their heads are marked in a bit per item, and the
// pop-count up to an item is its bucket.  Scattered stores bound the kernel: those of a table go to
// its strip of 4 n bytes, tiles in table order, which the L2 merges into full lines.  (A thread per
// bucket that walks the bucket's rows waits for one load after another: 11.6 ms at 10M x 48.)
__global__ void __launch_bounds__(IB_THREADS)
bucket_bounds_kernel(const int32_t* __restrict__ bucket_offsets, const int32_t* __restrict__ cand, int n, int t0,
                     int tiles_per_table, const uint32_t* __restrict__ tile_base, PackedBounds pb,
                     bool pairs, uint32_t* __restrict__ packed) {
    constexpr int WORDS = IB_TILE / 32;
    __shared__ int32_t s_off[IB_TILE + 2];  // [0] the bucket before the tile's first head, then its heads, then the next head
    __shared__ uint32_t s_bits[WORDS];
    __shared__ uint32_t s_pref[WORDS];
    const int table = blockIdx.x / tiles_per_table, t = t0 + table;
    const int lt = blockIdx.x - table * tiles_per_table;
    const int tile = t * tiles_per_table + lt;
    const int tbase = t * n;
    const int first = tbase + lt * IB_TILE, count = min(IB_TILE, n - lt * IB_TILE);
    const int lane = threadIdx.x & 31;
    int32_t row[IB_IPT];
#pragma unroll
    for (int i = 0; i < IB_IPT; ++i) {
        const int local = i * IB_THREADS + threadIdx.x;
        row[i] = local < count ? cand[first + local] : 0;
    }
    const int b0 = (int)tile_base[tile], heads = (int)tile_base[tile + 1] - b0;
    if (threadIdx.x < WORDS) s_bits[threadIdx.x] = 0;
    for (int j = threadIdx.x; j < heads + 2; j += IB_THREADS) s_off[j] = b0 - 1 + j >= 0 ? bucket_offsets[b0 - 1 + j] : 0;
    __syncthreads();
    for (int j = 1 + threadIdx.x; j <= heads; j += IB_THREADS) {
        const int local = s_off[j] - first;
        atomicOr(&s_bits[local >> 5], 1u << (local & 31));
    }
    __syncthreads();
    if (threadIdx.x < 32) {
        uint32_t run = 0;
        for (int w0 = 0; w0 < WORDS; w0 += 32) {
            const uint32_t c = __popc(s_bits[w0 + lane]);
            uint32_t inc = c;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t x = __shfl_up_sync(0xFFFFFFFFu, inc, o);
                if (lane >= o) inc += x;
            }
            s_pref[w0 + lane] = run + inc - c;
            run += __shfl_sync(0xFFFFFFFFu, inc, 31);
        }
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < IB_IPT; ++i) {
        const int local = i * IB_THREADS + threadIdx.x;
        if (local >= count) continue;
        const int j = (int)(s_pref[local >> 5] + __popc(s_bits[local >> 5] & (0xFFFFFFFFu >> (31 - lane))));
        const int lo = s_off[j], hi = s_off[j + 1];
        if (hi - lo > 1) {
            uint32_t word = (uint32_t)(lo - tbase) | (min((uint32_t)(hi - lo), pb.max_len) << pb.pos_bits);
            if (pairs && hi - lo == 2) word = PB_PAIR | (uint32_t)cand[lo == first + local ? hi - 1 : lo];
            packed[(size_t)tbase + row[i]] = word;
        }
    }
}

// The lists of a set of queries: an array of [x, y) per (table, query), table major, or the packed
// form of a self-join.
struct BoundsView {
    const int2* pair;                // or null: packed
    const uint32_t* packed;
    const int32_t* bucket_offsets;   // packed: to find the end of a list that is too long for its word
    const int32_t* table_offsets;
    PackedBounds pb;
    int n_q;                         // queries (a self-join: rows)
    __device__ __forceinline__ int2 get(int t, int q) const {
        if (pair) return pair[(size_t)t * n_q + q];
        return unpack(t, packed[(size_t)t * n_q + q]);
    }
    // not for PB_PAIR words
    __device__ __forceinline__ int2 unpack(int t, uint32_t w) const {
        if (w == 0) return make_int2(0, 0);
        const int lo = t * n_q + (int)(w & ((1u << pb.pos_bits) - 1u));
        const uint32_t len = w >> pb.pos_bits;
        if (len < pb.max_len) return make_int2(lo, lo + (int)len);
        int a = table_offsets[t], b = table_offsets[t + 1] - 1;  // the bucket that starts at lo
        while (a < b) {
            const int mid = a + ((b - a) >> 1);
            if (bucket_offsets[mid] < lo) a = mid + 1; else b = mid;
        }
        return make_int2(lo, bucket_offsets[a + 1]);
    }
};

#define CULSH_DISPATCH_NW(NWVAL, ...)                                         \
    switch (NWVAL) {                                                          \
        case 1: { constexpr int NW = 1; __VA_ARGS__; } break;                 \
        case 2: { constexpr int NW = 2; __VA_ARGS__; } break;                 \
        case 4: { constexpr int NW = 4; __VA_ARGS__; } break;                 \
        case 8: { constexpr int NW = 8; __VA_ARGS__; } break;                 \
        case 16: { constexpr int NW = 16; __VA_ARGS__; } break;               \
        default: ::culsh_b200::fail(CULSH_ERR_UNSUPPORTED, "unsupported key width"); \
    }

// ---------------------------------------------------------------------------------------
// Conversions between packed keys and upstream's raw signature bytes.
// ---------------------------------------------------------------------------------------
// raw: [count][sig_nbytes] (uint8 0/1 per hash, or little-endian int32/uint32 per hash)
__global__ void unpack_keys_kernel(const uint32_t* __restrict__ keys, size_t count, int family,
                                   int k, int NW, int elem_bytes, uint8_t* __restrict__ raw) {
    size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= count) return;
    const uint32_t* key = keys + i * NW;
    if (family == CULSH_RPLSH) {
        uint8_t* dst = raw + i * k;
        for (int j = 0; j < k; ++j) {
            int pos = k - 1 - j;
            dst[j] = (uint8_t)((key[NW - 1 - (pos >> 5)] >> (pos & 31)) & 1u);
        }
    } else {
        int32_t* dst = reinterpret_cast<int32_t*>(raw + i * (size_t)k * 4);
        const int pad = NW * 4 - k * elem_bytes;
        for (int j = 0; j < k; ++j) {
            uint32_t v = 0;
            for (int c = 0; c < elem_bytes; ++c) {
                int bp = pad + j * elem_bytes + c;  // big-endian byte position in the key
                uint32_t byte = (key[bp >> 2] >> (24 - 8 * (bp & 3))) & 0xFFu;
                v |= byte << (8 * c);
            }
            if (family == CULSH_PSLSH && elem_bytes < 4) {  // sign-extend
                int sh = 32 - 8 * elem_bytes;
                v = (uint32_t)(((int32_t)(v << sh)) >> sh);
            }
            dst[j] = (int32_t)v;
        }
    }
}

// Largest |value| bucket of raw int32 signatures needs: 1, 2 or 4 bytes (p-stable load).
__global__ void pslsh_width_kernel(const int32_t* __restrict__ raw, size_t count, int* __restrict__ width) {
    size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    int w = 1;
    if (i < count) {
        int v = raw[i];
        if (v < -32768 || v > 32767) w = 4;
        else if (v < -128 || v > 127) w = 2;
    }
    w = max(w, __shfl_xor_sync(0xFFFFFFFFu, w, 16));
    w = max(w, __shfl_xor_sync(0xFFFFFFFFu, w, 8));
    w = max(w, __shfl_xor_sync(0xFFFFFFFFu, w, 4));
    w = max(w, __shfl_xor_sync(0xFFFFFFFFu, w, 2));
    w = max(w, __shfl_xor_sync(0xFFFFFFFFu, w, 1));
    if ((threadIdx.x & 31) == 0 && w > 1) atomicMax(width, w);
}

__global__ void pack_keys_kernel(const uint8_t* __restrict__ raw, size_t count, int family, int k,
                                 int NW, int elem_bytes, uint32_t* __restrict__ keys) {
    size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= count) return;
    uint32_t* key = keys + i * NW;
    for (int w = 0; w < NW; ++w) key[w] = 0;
    if (family == CULSH_RPLSH) {
        const uint8_t* src = raw + i * k;
        for (int j = 0; j < k; ++j) {
            int pos = k - 1 - j;
            if (src[j]) key[NW - 1 - (pos >> 5)] |= 1u << (pos & 31);
        }
    } else {
        const uint32_t* src = reinterpret_cast<const uint32_t*>(raw + i * (size_t)k * 4);
        const int pad = NW * 4 - k * elem_bytes;
        for (int j = 0; j < k; ++j) {
            uint32_t v = src[j];
            for (int c = 0; c < elem_bytes; ++c) {
                int bp = pad + j * elem_bytes + c;
                key[bp >> 2] |= ((v >> (8 * c)) & 0xFFu) << (24 - 8 * (bp & 3));
            }
        }
    }
}

// Packed key of every indexed row, in row order: out[(t * n + row) * NW + w] = key of the bucket
// that holds `row` in table t.  One thread per bucket walks the bucket's rows (buckets of an LSH
// index are short); the stores of a table stay inside its n * NW words.
template <int NW>
__global__ void __launch_bounds__(256)
row_keys_kernel(const uint32_t* __restrict__ bucket_keys, const int32_t* __restrict__ bucket_offsets,
                const int32_t* __restrict__ cand, int n_buckets, int n, uint32_t* __restrict__ out) {
    const int b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= n_buckets) return;
    uint32_t key[NW];
#pragma unroll
    for (int w = 0; w < NW; ++w) key[w] = bucket_keys[(size_t)b * NW + w];
    const int lo = bucket_offsets[b], hi = bucket_offsets[b + 1];
    if (lo >= hi) return;
    const size_t table_base = (size_t)(lo / n) * (size_t)n;  // a bucket lies inside one table
    for (int p = lo; p < hi; ++p) {
        uint32_t* dst = out + (table_base + (size_t)cand[p]) * NW;
#pragma unroll
        for (int w = 0; w < NW; ++w) dst[w] = key[w];
    }
}

}  // namespace culsh_b200
