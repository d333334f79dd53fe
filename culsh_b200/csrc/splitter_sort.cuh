// Sort of a table's (key, row id) pairs by sampled splitters: the rows go into bins of about a thousand, a bin
// is sorted by one CTA in shared memory.  It takes keys that a radix sort would need many passes for - seven bytes and more, up to SS_CAP
// rows all of two words and more - in tables that a CTA or a cluster does not sort faster as a whole, and that are not too long: see sort_by_splitters.
//
//   1. splitter_sample_kernel   sorts SS_OVER rows a bin and more, drawn from all of the table, SS_CAP a CTA
//      splitter_rank_kernel     (tables of several such chunks) ranks the samples among all of the table's
//   2. splitter_classify_kernel finds the bin of every row among the splitters, and counts the rows of each tile in each bin
//   3. splitter_scan_kernel     counts of the tiles before a tile
//   4. splitter_scatter_kernel  writes the row ids, bin after bin
//   5. splitter_short_bin_kernel (keys of up to four words), splitter_bin_kernel
//                               gather the keys of a bin, sort them and write keys and ids
//
// The order is that of (key, row id), so no two rows are alike and bins stay even however often a key repeats; what
// the order of equal keys is does not depend on the order in which a CTA's rows arrive.  How full a bin is, is a matter of
// the sample: one of more than SS_CAP rows is sorted in pieces, which are brought together by rank.
#pragma once

#include "common.cuh"
#include "radix_sort.cuh"

namespace culsh_b200 {

constexpr int SS_THREADS = 256;
constexpr int SS_ITEMS = 8;                     // of a thread, next to one another in the order
constexpr int SS_CAP = SS_THREADS * SS_ITEMS;   // rows that a CTA sorts at once
constexpr int SS_BIN_ROWS = 1024;               // rows of a bin on average, at most
constexpr int SS_OVER = 8;                      // samples for each bin, at least
constexpr int SS_MAX_BINS = 4096;
constexpr int SS_TILE = 16384, SS_SHORT_TILE = 4096;  // rows of a CTA that classifies or scatters, and where these would be few, at least
constexpr int SS_TILE_THREADS = 512;

inline int splitter_bins(int n) {
    int bins = 1;
    if (n <= SS_CAP) return bins;
    while ((int64_t)bins * SS_BIN_ROWS < n) bins *= 2;
    return bins;
}

// A key in 64-bit parts, the most significant first, which compare as the key does: all of it up to four words, the first four words in
// use of longer ones, whose rest is read again where these are the same.
template <int NW>
struct KeyParts {
    uint64_t p[2];
};

template <int NW>
__device__ __forceinline__ KeyParts<NW> key_parts(const uint32_t* __restrict__ key, int skip /* leading words that are zero in all keys */) {
    KeyParts<NW> k;
    if constexpr (NW == 2) {
        const uint2 v = *reinterpret_cast<const uint2*>(key);
        k.p[0] = 0;
        k.p[1] = (uint64_t)v.x << 32 | v.y;
    } else if constexpr (NW == 4) {
        const uint4 v = *reinterpret_cast<const uint4*>(key);
        k.p[0] = (uint64_t)v.x << 32 | v.y;
        k.p[1] = (uint64_t)v.z << 32 | v.w;
    } else {
        key += skip;
        k.p[0] = (uint64_t)key[0] << 32 | key[1];
        k.p[1] = (uint64_t)key[2] << 32 | key[3];
    }
    return k;
}

// The order of two keys whose parts are the same, by the words behind them, in whole fours that are read together.
template <int NW>
__device__ __forceinline__ int compare_rest(const uint32_t* __restrict__ ka, const uint32_t* __restrict__ kb, int skip) {
    int c = 0;
#pragma unroll
    for (int q = NW / 4 - 1; q >= 1; --q) {
        if (4 * q < skip + 1) continue;  // nothing behind the parts
        const uint4 x = reinterpret_cast<const uint4*>(ka)[q], y = reinterpret_cast<const uint4*>(kb)[q];
        const uint64_t x0 = (uint64_t)x.x << 32 | x.y, x1 = (uint64_t)x.z << 32 | x.w, y0 = (uint64_t)y.x << 32 | y.y, y1 = (uint64_t)y.z << 32 | y.w;
        if (x1 != y1) c = x1 < y1 ? -1 : 1;
        if (x0 != y0) c = x0 < y0 ? -1 : 1;
    }
    return c;
}

// Whether row a comes before row b, whose parts are the same.  SS_NONE is no row and comes last.
constexpr uint32_t SS_NONE = 0xFFFFFFFFu;
template <int NW>
__device__ __forceinline__ bool tie_less(const uint32_t* __restrict__ table, int skip, uint32_t a, uint32_t b) {
    if constexpr (NW > 4) {
        if (a != SS_NONE && b != SS_NONE) {
            const int c = compare_rest<NW>(table + (size_t)a * NW, table + (size_t)b * NW, skip);
            if (c != 0) return c < 0;
        }
    }
    return a < b;
}
template <int NW>
__device__ __forceinline__ bool row_less(const uint32_t* __restrict__ table, int skip, const KeyParts<NW>& ka, uint32_t a, const KeyParts<NW>& kb,
                                         uint32_t b) {
    if (ka.p[0] != kb.p[0]) return ka.p[0] < kb.p[0];
    if (ka.p[1] != kb.p[1]) return ka.p[1] < kb.p[1];
    return tie_less<NW>(table, skip, a, b);
}

// A row id and W words of a key as one number.
template <int W>
struct BinItem {
    uint32_t w[W + 1];  // the row id, then the words of the key, the least significant first
};
template <int W>
__device__ __forceinline__ bool item_less(const BinItem<W>& a, const BinItem<W>& b) {
    uint32_t m = 0;  // the borrow of a - b
    if constexpr (W == 0) {
        m = a.w[0] < b.w[0];
    } else if constexpr (W == 1) {
        asm("{\n\t.reg .u32 t;\n\tsub.cc.u32 t, %1, %3;\n\tsubc.cc.u32 t, %2, %4;\n\tsubc.u32 %0, 0, 0;\n\t}"
            : "=r"(m) : "r"(a.w[0]), "r"(a.w[1]), "r"(b.w[0]), "r"(b.w[1]));
    } else if constexpr (W == 2) {
        asm("{\n\t.reg .u32 t;\n\tsub.cc.u32 t, %1, %4;\n\tsubc.cc.u32 t, %2, %5;\n\tsubc.cc.u32 t, %3, %6;\n\tsubc.u32 %0, 0, 0;\n\t}"
            : "=r"(m) : "r"(a.w[0]), "r"(a.w[1]), "r"(a.w[2]), "r"(b.w[0]), "r"(b.w[1]), "r"(b.w[2]));
    } else if constexpr (W == 3) {
        asm("{\n\t.reg .u32 t;\n\tsub.cc.u32 t, %1, %5;\n\tsubc.cc.u32 t, %2, %6;\n\tsubc.cc.u32 t, %3, %7;\n\tsubc.cc.u32 t, %4, %8;\n\t"
            "subc.u32 %0, 0, 0;\n\t}"
            : "=r"(m) : "r"(a.w[0]), "r"(a.w[1]), "r"(a.w[2]), "r"(a.w[3]), "r"(b.w[0]), "r"(b.w[1]), "r"(b.w[2]), "r"(b.w[3]));
    } else {
        asm("{\n\t.reg .u32 t;\n\tsub.cc.u32 t, %1, %6;\n\tsubc.cc.u32 t, %2, %7;\n\tsubc.cc.u32 t, %3, %8;\n\tsubc.cc.u32 t, %4, %9;\n\t"
            "subc.cc.u32 t, %5, %10;\n\tsubc.u32 %0, 0, 0;\n\t}"
            : "=r"(m) : "r"(a.w[0]), "r"(a.w[1]), "r"(a.w[2]), "r"(a.w[3]), "r"(a.w[4]), "r"(b.w[0]), "r"(b.w[1]), "r"(b.w[2]), "r"(b.w[3]), "r"(b.w[4]));
    }
    return m != 0;
}
// ---------------------------------------------------------------------------------------
// Merge sort of up to SS_CAP rows by one CTA.  The parts and ids stay where they are, 16-bit positions are what moves: a thread
// sorts SS_ITEMS of them in registers, then runs of twice the length come from two, a thread writing SS_ITEMS places of the result
// from where a search along its diagonal says.  Only the first part of a key is read as a rule.  Words behind the parts come from memory, one comparison
// after the other, which is most of the time where many keys are the same: rows that are all alike need no look at them, and others read them in whole
// fours.  8 tables of 300,000 keys, word by word and this way, the whole sort: 32 bytes, alike 1,090 and 409 us (by radix passes 845), ten different ones 1,195 and
// 456 (947), 7,500 groups of near duplicates 735 and 546 (990), all different 276 and 270 (1,013); 64 bytes, alike 3,006 and 577 (1,976).
// ---------------------------------------------------------------------------------------
template <int NW>
struct BlockSort {
    struct Smem {
        uint64_t p[2][SS_CAP];
        uint32_t id[SS_CAP];
        uint16_t ord[2][SS_CAP];
    };
    Smem& s;
    const uint32_t* table;
    int skip;
    bool rest;  // whether the words behind the parts tell rows apart

    // Row `row`, whose parts are k, into place i; whether its key is that of row `first`, whose parts are k_first.
    static __device__ __forceinline__ bool put(Smem& s, const uint32_t* table, int skip, int i, uint32_t row, uint32_t first, const KeyParts<NW>& k_first) {
        const KeyParts<NW> k = key_parts<NW>(table + (size_t)row * NW, skip);
        s.p[0][i] = k.p[0];
        s.p[1][i] = k.p[1];
        s.id[i] = row;
        if constexpr (NW > 4)
            return k.p[0] == k_first.p[0] && k.p[1] == k_first.p[1] && compare_rest<NW>(table + (size_t)row * NW, table + (size_t)first * NW, skip) == 0;
        return true;
    }

    __device__ __forceinline__ bool less(uint64_t pa, uint32_t a, uint64_t pb, uint32_t b) const {
        if (pa != pb) return pa < pb;
        const uint64_t qa = s.p[1][a], qb = s.p[1][b];
        if (qa != qb) return qa < qb;
        return rest ? tie_less<NW>(table, skip, s.id[a], s.id[b]) : s.id[a] < s.id[b];
    }

    // Sorts the m rows whose parts and ids are in `s`; the positions in order.  Called by all threads, behind a barrier.
    __device__ const uint16_t* sort(int m) const {
        const int tid = threadIdx.x, at = tid * SS_ITEMS;
        const int padded = (m + SS_ITEMS - 1) / SS_ITEMS * SS_ITEMS;
        if (tid < padded - m) {  // up to a whole thread's items: rows that come last
            s.p[0][m + tid] = s.p[1][m + tid] = ~0ull;
            s.id[m + tid] = SS_NONE;
        }
        __syncthreads();
        const bool on = at < padded;
        if (on) {
            uint64_t p[SS_ITEMS];
            uint32_t x[SS_ITEMS];
#pragma unroll
            for (int i = 0; i < SS_ITEMS; ++i) {
                p[i] = s.p[0][at + i];
                x[i] = at + i;
            }
            auto order = [&](int i, int j) {
                if (less(p[j], x[j], p[i], x[i])) {
                    const uint64_t q = p[i];
                    const uint32_t y = x[i];
                    p[i] = p[j]; x[i] = x[j];
                    p[j] = q; x[j] = y;
                }
            };
            // Batcher's odd-even merge sort of eight
            order(0, 1); order(2, 3); order(4, 5); order(6, 7);
            order(0, 2); order(1, 3); order(4, 6); order(5, 7);
            order(1, 2); order(5, 6);
            order(0, 4); order(1, 5); order(2, 6); order(3, 7);
            order(2, 4); order(3, 5);
            order(1, 2); order(3, 4); order(5, 6);
            *reinterpret_cast<uint4*>(s.ord[0] + at) = make_uint4(x[0] | x[1] << 16, x[2] | x[3] << 16, x[4] | x[5] << 16, x[6] | x[7] << 16);
        }
        __syncthreads();
        int cur = 0;
        for (int run = SS_ITEMS; run < padded; run *= 2, cur ^= 1) {
            if (on) {
                const uint16_t* from = s.ord[cur];
                const int base = at & ~(2 * run - 1);
                const int ea = min(base + run, padded), eb = min(base + 2 * run, padded);
                const int d = at - base;
                int lo = max(0, d - (eb - ea)), hi = min(d, ea - base);
                while (lo < hi) {  // how many of the first run come before this thread's places
                    const int mid = (lo + hi) >> 1;
                    const uint32_t a = from[base + mid], b = from[ea + d - 1 - mid];
                    if (less(s.p[0][b], b, s.p[0][a], a)) hi = mid;
                    else lo = mid + 1;
                }
                int ia = base + lo, ib = ea + d - lo;
                uint32_t a = ia < ea ? from[ia] : 0u, b = ib < eb ? from[ib] : 0u;
                uint64_t pa = s.p[0][a], pb = s.p[0][b];
                uint32_t out[SS_ITEMS];
#pragma unroll
                for (int i = 0; i < SS_ITEMS; ++i) {
                    const bool first = ia < ea && (ib >= eb || !less(pb, b, pa, a));
                    out[i] = first ? a : b;
                    const int next = first ? ++ia : ++ib;
                    if (next < (first ? ea : eb)) {
                        const uint32_t x = from[next];
                        const uint64_t p = s.p[0][x];
                        if (first) { a = x; pa = p; }
                        else { b = x; pb = p; }
                    }
                }
                *reinterpret_cast<uint4*>(s.ord[cur ^ 1] + at) =
                    make_uint4(out[0] | out[1] << 16, out[2] | out[3] << 16, out[4] | out[5] << 16, out[6] | out[7] << 16);
            }
            __syncthreads();
        }
        return s.ord[cur];
    }
};

// ---------------------------------------------------------------------------------------
// Splitters
// ---------------------------------------------------------------------------------------
// Sorted rows with their parts: the samples of a table, chunk after chunk, or its splitters.
template <int NW>
struct RowList {
    uint64_t* p[2];
    uint32_t* id;
    __device__ __forceinline__ KeyParts<NW> parts(size_t i) const {
        return KeyParts<NW>{{p[0][i], p[1][i]}};
    }
    __device__ __forceinline__ void put(size_t i, const KeyParts<NW>& k, uint32_t row) const {
        p[0][i] = k.p[0];
        p[1][i] = k.p[1];
        id[i] = row;
    }
};

// A CTA for each (table, chunk of SS_CAP samples).  Sample i is a row of the i-th of `samples` equal stretches of the table, which of
// them is scrambled: rows that repeat with some period are sampled like any others.
template <int NW>
__global__ void __launch_bounds__(SS_THREADS)
splitter_sample_kernel(const uint32_t* __restrict__ keys, int n, int skip, int samples, int chunks, int bins, int over,
                       RowList<NW> sorted /* one chunk: the splitters */, KernelBefore kernel_before) {
    behind_kernel_before(keys, kernel_before);
    extern __shared__ __align__(16) unsigned char ss_smem[];
    using Sort = BlockSort<NW>;
    auto& s = *reinterpret_cast<typename Sort::Smem*>(ss_smem);
    const int t = blockIdx.x / chunks, chunk = blockIdx.x - t * chunks;
    const uint32_t* table = keys + (size_t)t * n * NW;
    const int m = min(SS_CAP, samples - chunk * SS_CAP);
    const KeyParts<NW> first = key_parts<NW>(table, skip);
    bool alike = true;
    for (int i = threadIdx.x; i < m; i += SS_THREADS) {
        const uint32_t g = (uint32_t)(chunk * SS_CAP + i);
        const uint32_t r0 = (uint32_t)((uint64_t)g * n / samples), r1 = (uint32_t)((uint64_t)(g + 1) * n / samples);
        uint32_t h = (g + 1u) * 0x9E3779B9u;  // mixed by the last steps of MurmurHash3
        h ^= h >> 16; h *= 0x85EBCA6Bu; h ^= h >> 13; h *= 0xC2B2AE35u; h ^= h >> 16;
        alike = Sort::put(s, table, skip, i, r0 + h % (r1 - r0), 0u, first) && alike;
    }
    const bool rest = !__syncthreads_and(alike);
    const uint16_t* ord = Sort{s, table, skip, rest}.sort(m);
    for (int i = threadIdx.x; i < m; i += SS_THREADS) {
        const uint32_t x = ord[i];
        const KeyParts<NW> k{{s.p[0][x], s.p[1][x]}};
        if (chunks > 1) sorted.put((size_t)blockIdx.x * SS_CAP + i, k, s.id[x]);
        else if (i > 0 && i % over == 0) sorted.put((size_t)t * bins + i / over - 1, k, s.id[x]);
    }
}

// A thread for each sample: its rank among the table's samples.  Every SS_OVER-th becomes a splitter.  samples = chunks * SS_CAP.
template <int NW>
__global__ void __launch_bounds__(256)
splitter_rank_kernel(const uint32_t* __restrict__ keys, int n, int skip, int chunks, int bins, int total, RowList<NW> sorted, RowList<NW> splitters, KernelBefore kernel_before) {
    behind_kernel_before(keys, kernel_before);
    const int i = blockIdx.x * 256 + threadIdx.x;
    if (i >= total) return;
    const int samples = chunks * SS_CAP, t = i / samples, own = (i - t * samples) / SS_CAP;
    const uint32_t* table = keys + (size_t)t * n * NW;
    const KeyParts<NW> k = sorted.parts(i);
    const uint32_t row = sorted.id[i];
    int rank = (i - t * samples) % SS_CAP;
    for (int c = 0; c < chunks; ++c) {
        if (c == own) continue;
        const size_t first = (size_t)t * samples + (size_t)c * SS_CAP;
        int at = 0;  // samples of that chunk before this one
#pragma unroll
        for (int step = SS_CAP / 2; step > 0; step >>= 1)
            if (row_less<NW>(table, skip, sorted.parts(first + at + step - 1), sorted.id[first + at + step - 1], k, row)) at += step;
        if (row_less<NW>(table, skip, sorted.parts(first + at), sorted.id[first + at], k, row)) ++at;
        rank += at;
    }
    if (rank > 0 && rank % SS_OVER == 0) splitters.put((size_t)t * bins + rank / SS_OVER - 1, k, row);
}

// ---------------------------------------------------------------------------------------
// Rows into bins
// ---------------------------------------------------------------------------------------
inline size_t splitter_classify_smem(int bins) { return (size_t)bins * (16 + 8 + 4 + 4); }

// A CTA for each tile.  bin_of[t * n + row]; tile_hist [table][tile][bin].  Bound by the reads of the splitters from shared memory, and the wider
// one is the more lanes get in one another's way: a row is searched by one word of its key after the other, among the splitters
// that agree in those before.  2M rows x 32 tables: over whole keys 2,470 us, over halves 1,520, over words 1,194.
template <int NW>
__global__ void __launch_bounds__(SS_TILE_THREADS)
splitter_classify_kernel(const uint32_t* __restrict__ keys, int n, int skip, int tile, int tiles, int bins, RowList<NW> splitters,
                         uint16_t* __restrict__ bin_of, uint32_t* __restrict__ tile_hist) {
    extern __shared__ __align__(16) unsigned char ss_smem[];
    uint32_t* s_word = reinterpret_cast<uint32_t*>(ss_smem);                    // [4][bins] words of the splitters, the most significant first
    uint32_t* s_id = s_word + 4 * (size_t)bins;                                 // [bins]
    uint32_t* s_hist = s_id + bins;                                             // [bins]
    uint16_t* s_end = reinterpret_cast<uint16_t*>(s_hist + bins);               // [4][bins] end of those that agree with one in this word and all before
    const int tid = threadIdx.x, last = bins - 1;                               // splitters
    const int t = blockIdx.x / tiles, lt = blockIdx.x - t * tiles;
    const int row0 = lt * tile, count = min(tile, n - row0);
    const uint32_t* table = keys + (size_t)t * n * NW;
    for (int i = tid; i < bins; i += SS_TILE_THREADS) {
        if (i < last) {
            const KeyParts<NW> k = splitters.parts((size_t)t * bins + i);
            s_word[i] = (uint32_t)(k.p[0] >> 32);
            s_word[bins + i] = (uint32_t)k.p[0];
            s_word[2 * bins + i] = (uint32_t)(k.p[1] >> 32);
            s_word[3 * bins + i] = (uint32_t)k.p[1];
            s_id[i] = splitters.id[(size_t)t * bins + i];
        }
        s_hist[i] = 0;
    }
    __syncthreads();
    for (int i = tid; i < last; i += SS_TILE_THREADS) {
        int end = last;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const uint32_t x = s_word[j * bins + i];
            int lo = i + 1, hi = end;
            while (lo < hi) {
                const int mid = (lo + hi) >> 1;
                if (s_word[j * bins + mid] == x) lo = mid + 1;
                else hi = mid;
            }
            end = lo;
            s_end[j * bins + i] = (uint16_t)end;
        }
    }
    __syncthreads();
    constexpr int LOADS = 4, FIRST = NW == 2 ? 2 : 0;
    auto word = [](const KeyParts<NW>& k, int w) { return (uint32_t)(k.p[w >> 1] >> ((w & 1) ? 0 : 32)); };
    for (int i0 = tid; i0 < count; i0 += SS_TILE_THREADS * LOADS) {
        KeyParts<NW> k[LOADS];
        int at[LOADS];
#pragma unroll
        for (int j = 0; j < LOADS; ++j) {
            const int row = row0 + min(i0 + j * SS_TILE_THREADS, count - 1);
            k[j] = key_parts<NW>(table + (size_t)row * NW, skip);
            at[j] = 0;
        }
        for (int step = bins >> 1; step > 0; step >>= 1) {  // splitters whose first word is below the row's
#pragma unroll
            for (int j = 0; j < LOADS; ++j)
                if (s_word[FIRST * bins + at[j] + step - 1] < word(k[j], FIRST)) at[j] += step;
        }
#pragma unroll
        for (int j = 0; j < LOADS; ++j) {
            const int i = i0 + j * SS_TILE_THREADS;
            const uint32_t row = (uint32_t)(row0 + min(i, count - 1));
            int lo = at[j];
            uint32_t x = word(k[j], FIRST);
            for (int w = FIRST; lo < last && s_word[w * bins + lo] == x; ) {  // the splitters from lo to the end of its run agree with the row so far
                int hi = s_end[w * bins + lo];
                const int end = hi;
                if (++w == 4) {
                    while (lo < hi) {
                        const int mid = (lo + hi) >> 1;
                        if (tie_less<NW>(table, skip, row, s_id[mid])) hi = mid;
                        else lo = mid + 1;
                    }
                    break;
                }
                x = word(k[j], w);
                while (lo < hi) {
                    const int mid = (lo + hi) >> 1;
                    if (s_word[w * bins + mid] < x) lo = mid + 1;
                    else hi = mid;
                }
                if (lo == end) break;
            }
            if (i < count) {
                bin_of[(size_t)t * n + row0 + i] = (uint16_t)lo;
                atomicAdd(&s_hist[lo], 1u);
            }
        }
    }
    __syncthreads();
    for (int i = tid; i < bins; i += SS_TILE_THREADS) tile_hist[(size_t)blockIdx.x * bins + i] = s_hist[i];
}

// A thread for each (table, bin): its counts become those of the tiles before, and bin_total theirs.
constexpr int SS_SCAN_THREADS = 64;
__global__ void __launch_bounds__(SS_SCAN_THREADS)
splitter_scan_kernel(uint32_t* __restrict__ tile_hist, int tiles, int bins, int total, uint32_t* __restrict__ bin_total, KernelBefore kernel_before) {
    behind_kernel_before(tile_hist, bin_total, kernel_before);
    const int i = blockIdx.x * SS_SCAN_THREADS + threadIdx.x;
    if (i >= total) return;
    const int t = i / bins, b = i - t * bins;
    uint32_t* h = tile_hist + (size_t)t * tiles * bins + b;
    uint32_t run = 0;
    constexpr int LOADS = 16;
    for (int lt = 0; lt < tiles; lt += LOADS) {
        uint32_t x[LOADS];
#pragma unroll
        for (int j = 0; j < LOADS; ++j) x[j] = lt + j < tiles ? h[(size_t)(lt + j) * bins] : 0u;
#pragma unroll
        for (int j = 0; j < LOADS; ++j) {
            if (lt + j < tiles) h[(size_t)(lt + j) * bins] = run;
            run += x[j];
        }
    }
    bin_total[i] = run;
}

inline size_t splitter_scatter_smem(int tile, int bins) { return (size_t)tile * 4 + (size_t)bins * 8; }

// A CTA for each tile: its rows in the order of their bins through shared memory, out in runs.  The first tile of a table leaves where its
// bins start in bin_start[t * (bins + 1) ...].
__global__ void __launch_bounds__(SS_TILE_THREADS)
splitter_scatter_kernel(const uint16_t* __restrict__ bin_of, int n, int tile, int tiles, int bins, const uint32_t* __restrict__ tile_hist,
                        const uint32_t* __restrict__ bin_total, uint32_t* __restrict__ bin_start,
                        uint32_t* __restrict__ ids, KernelBefore kernel_before) {
    behind_kernel_before(bin_of, tile_hist, bin_total, bin_start, ids, kernel_before);
    extern __shared__ __align__(16) unsigned char ss_smem[];
    uint16_t* s_row = reinterpret_cast<uint16_t*>(ss_smem);            // [tile] its rows, bin after bin
    uint16_t* s_bin = s_row + tile;                                    // [tile] their bins
    uint32_t* s_cur = reinterpret_cast<uint32_t*>(s_bin + tile);       // [bins] next place of a bin inside the tile
    uint32_t* s_dst = s_cur + bins;                                    // [bins] place in `ids` of the tile's place 0
    __shared__ uint32_t s_warp[2][SS_TILE_THREADS / 32];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int t = blockIdx.x / tiles, lt = blockIdx.x - t * tiles;
    const int row0 = lt * tile, count = min(tile, n - row0);
    const uint32_t *before = tile_hist + (size_t)blockIdx.x * bins, *total = bin_total + (size_t)t * bins;
    const uint32_t* behind = lt + 1 < tiles ? before + bins : total;
    uint32_t base_here = 0, base_all = 0;  // of the bins of the steps before
    for (int b0 = 0; b0 < bins; b0 += SS_TILE_THREADS) {
        const int b = b0 + tid;
        const uint32_t first = b < bins ? before[b] : 0u, here = b < bins ? behind[b] - first : 0u, all = b < bins ? total[b] : 0u;
        uint32_t x = here, y = all;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t u = __shfl_up_sync(0xFFFFFFFFu, x, o), v = __shfl_up_sync(0xFFFFFFFFu, y, o);
            if (lane >= o) { x += u; y += v; }
        }
        __syncthreads();
        if (lane == 31) { s_warp[0][warp] = x; s_warp[1][warp] = y; }
        __syncthreads();
        uint32_t bx = base_here, by = base_all;
        for (int w = 0; w < SS_TILE_THREADS / 32; ++w) {
            const uint32_t u = s_warp[0][w], v = s_warp[1][w];
            if (w < warp) { bx += u; by += v; }
            base_here += u;
            base_all += v;
        }
        if (b < bins) {
            const uint32_t at = bx + x - here, start = by + y - all;
            s_cur[b] = at;
            s_dst[b] = (uint32_t)((size_t)t * n) + start + first - at;
            if (lt == 0) bin_start[(size_t)t * (bins + 1) + b] = start;
        }
    }
    if (lt == 0 && tid == 0) bin_start[(size_t)t * (bins + 1) + bins] = (uint32_t)n;
    __syncthreads();
    constexpr int LOADS = 8;
    const uint16_t* mine = bin_of + (size_t)t * n + row0;
    for (int i0 = tid; i0 < count; i0 += SS_TILE_THREADS * LOADS) {
        uint16_t b[LOADS];
#pragma unroll
        for (int j = 0; j < LOADS; ++j) b[j] = i0 + j * SS_TILE_THREADS < count ? mine[i0 + j * SS_TILE_THREADS] : (uint16_t)0;
#pragma unroll
        for (int j = 0; j < LOADS; ++j) {
            const int i = i0 + j * SS_TILE_THREADS;
            if (i < count) {
                const uint32_t to = atomicAdd(&s_cur[b[j]], 1u);
                s_row[to] = (uint16_t)i;
                s_bin[to] = b[j];
            }
        }
    }
    __syncthreads();
    for (int i = tid; i < count; i += SS_TILE_THREADS) ids[s_dst[s_bin[i]] + (uint32_t)i] = (uint32_t)row0 + s_row[i];
}

// A bin that was sorted in pieces of SS_CAP: the place of a row is its place in its own piece and the number of rows before it in each of the others.
template <int NW>
__device__ void place_pieces(const uint32_t* __restrict__ table, int skip, const uint32_t* ids, int m, uint32_t* __restrict__ keys_out,
                             uint32_t* __restrict__ ids_out) {
    __syncthreads();
    for (int i = threadIdx.x; i < m; i += SS_THREADS) {
        const uint32_t row = ids[i];
        const KeyParts<NW> k = key_parts<NW>(table + (size_t)row * NW, skip);
        const int own = i / SS_CAP;
        int rank = i % SS_CAP;
        for (int c = 0; c * SS_CAP < m; ++c) {
            if (c == own) continue;
            int lo = c * SS_CAP, hi = min(m, lo + SS_CAP);
            while (lo < hi) {
                const int mid = (lo + hi) >> 1;
                const uint32_t other = ids[mid];
                if (row_less<NW>(table, skip, key_parts<NW>(table + (size_t)other * NW, skip), other, k, row)) lo = mid + 1;
                else hi = mid;
            }
            rank += lo - c * SS_CAP;
        }
        uint32_t kk[NW];
        load_key<NW>(table + (size_t)row * NW, kk);
        store_key<NW>(keys_out + (size_t)rank * NW, kk);
        ids_out[rank] = row;
    }
}

// ---------------------------------------------------------------------------------------
// Bins in order.  A CTA for each.  ids [table][n]: the rows of the bins, overwritten (null: a table is one bin of its rows 0 .. n - 1,
// at most SS_CAP); keys in row order, keys_out and ids_out in the order of (key, row).
// ---------------------------------------------------------------------------------------
template <int NW>
__global__ void __launch_bounds__(SS_THREADS, 4)
splitter_bin_kernel(const uint32_t* __restrict__ keys, int n, int skip, int bins, const uint32_t* __restrict__ bin_start,
                    uint32_t* ids, uint32_t* __restrict__ keys_out, uint32_t* __restrict__ ids_out) {
    extern __shared__ __align__(16) unsigned char ss_smem[];
    using Sort = BlockSort<NW>;
    auto& s = *reinterpret_cast<typename Sort::Smem*>(ss_smem);
    const int tid = threadIdx.x;
    const int t = blockIdx.x / bins, b = blockIdx.x - t * bins;
    const uint32_t first = ids ? bin_start[(size_t)t * (bins + 1) + b] : 0u;
    const int m_all = ids ? (int)(bin_start[(size_t)t * (bins + 1) + b + 1] - first) : n;
    const uint32_t* table = keys + (size_t)t * n * NW;
    const size_t base = (size_t)t * n + first;
    for (int c0 = 0; c0 < m_all; c0 += SS_CAP) {
        const int m = min(SS_CAP, m_all - c0);
        __syncthreads();  // the piece before is out
        const uint32_t row0 = ids ? ids[base + c0] : 0u;
        const KeyParts<NW> k0 = key_parts<NW>(table + (size_t)row0 * NW, skip);
        bool alike = true;
        for (int i = tid; i < m; i += SS_THREADS) alike = Sort::put(s, table, skip, i, ids ? ids[base + c0 + i] : (uint32_t)i, row0, k0) && alike;
        const bool rest = !__syncthreads_and(alike);  // all rows alike: their ids are what is left
        const uint16_t* ord = Sort{s, table, skip, rest}.sort(m);
        if (m_all > SS_CAP) {  // a piece: its rows in order where they were
            for (int i = tid; i < m; i += SS_THREADS) ids[base + c0 + i] = s.id[ord[i]];
            continue;
        }
        for (int i = tid; i < m; i += SS_THREADS) {
            const uint32_t x = ord[i], row = s.id[x];
            uint32_t* to = keys_out + (base + i) * NW;
            uint32_t k[NW];
            load_key<NW>(table + (size_t)row * NW, k);
            store_key<NW>(to, k);
            ids_out[base + i] = row;
        }
    }
    if (m_all > SS_CAP) place_pieces<NW>(table, skip, ids + base, m_all, keys_out + base * NW, ids_out + base);
}

// ---------------------------------------------------------------------------------------
// Bins of keys of two and four words in order.  The keys of a bin lie between two splitters: less the lower one they take W words or none, and
// with the row id behind them they are numbers of W + 1 words, no two alike.  A warp sorts 32 * SS_ITEMS of them in registers (the network of the
// candidate sets, see warp_sort_unique), runs of warps are merged in shared memory.  Issue (44 % of the slots) and the reads of shared memory (69 % of
// their pipe) bound it: 64M keys of 16 bytes in 2.56 ms, where a merge sort of 16-bit positions from eight items on took 3.58, merges from 32 and 64
// items on instead of 256 3.04 and 2.89, and the network through shared memory instead of the last merges 2.97.
// ---------------------------------------------------------------------------------------
template <int W>
__device__ __forceinline__ void item_order(BinItem<W>& a, BinItem<W>& b) {
    const bool swap = item_less<W>(b, a);
#pragma unroll
    for (int i = 0; i <= W; ++i) {
        const uint32_t x = a.w[i], y = b.w[i];
        a.w[i] = swap ? y : x;
        b.w[i] = swap ? x : y;
    }
}

constexpr int SS_WARP_ROWS = 32 * SS_ITEMS;

// SS_WARP_ROWS items, place SS_ITEMS * lane + e in v[e] of `lane`.
template <int W>
__device__ __forceinline__ void warp_sort_items(BinItem<W> (&v)[SS_ITEMS], int lane) {
    // Batcher's odd-even merge sort of a lane's eight
    auto order = [&](int i, int j) { item_order<W>(v[i], v[j]); };
    order(0, 1); order(2, 3); order(4, 5); order(6, 7);
    order(0, 2); order(1, 3); order(4, 6); order(5, 7);
    order(1, 2); order(5, 6);
    order(0, 4); order(1, 5); order(2, 6); order(3, 7);
    order(2, 4); order(3, 5);
    order(1, 2); order(3, 4); order(5, 6);
#pragma unroll 1
    for (int ksz = 2 * SS_ITEMS; ksz <= SS_WARP_ROWS; ksz <<= 1) {
        auto exchange = [&](int mask, bool reverse) {  // with the lane `mask` away, the smaller ones to the lower lane
            const bool low = (lane & (reverse ? (mask + 1) / 2 : mask)) == 0;
            BinItem<W> o[SS_ITEMS];
#pragma unroll
            for (int e = 0; e < SS_ITEMS; ++e)
#pragma unroll
                for (int i = 0; i <= W; ++i) o[e].w[i] = __shfl_xor_sync(0xFFFFFFFFu, v[reverse ? SS_ITEMS - 1 - e : e].w[i], mask);
#pragma unroll
            for (int e = 0; e < SS_ITEMS; ++e) {
                const bool take = item_less<W>(o[e], v[e]) == low;
#pragma unroll
                for (int i = 0; i <= W; ++i) v[e].w[i] = take ? o[e].w[i] : v[e].w[i];
            }
        };
        exchange(ksz / SS_ITEMS - 1, true);
#pragma unroll 1
        for (int j = ksz >> 2; j >= SS_ITEMS; j >>= 1) exchange(j / SS_ITEMS, false);
#pragma unroll
        for (int j = SS_ITEMS / 2; j > 0; j >>= 1)
#pragma unroll
            for (int e = 0; e < SS_ITEMS; ++e)
                if ((e & j) == 0) order(e, e | j);
    }
}

// Sorts the rows ids[0 .. m - 1] (null: 0 .. m - 1), m <= CAP, whose keys less `low` take W words with `shift` bits to spare, which the
// items do not have: their first word tells most of them apart.  s_w[i][place] is word i of an item on return, behind a barrier.  Called by all threads.
template <int NW, int W, int CAP>
__device__ __forceinline__ void sort_bin(const uint32_t* __restrict__ table, const uint32_t* ids, int m, const uint32_t (&low)[4],
                                         int shift, uint32_t (*s_w)[CAP]) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, at = tid * SS_ITEMS;
    const int padded = (m + SS_WARP_ROWS - 1) / SS_WARP_ROWS * SS_WARP_ROWS;
    const bool on = at < padded;  // whole warps
    auto store = [&](const BinItem<W> (&v)[SS_ITEMS]) {
#pragma unroll
        for (int i = 0; i <= W; ++i) {
            reinterpret_cast<uint4*>(s_w[i] + at)[0] = make_uint4(v[0].w[i], v[1].w[i], v[2].w[i], v[3].w[i]);
            reinterpret_cast<uint4*>(s_w[i] + at)[1] = make_uint4(v[4].w[i], v[5].w[i], v[6].w[i], v[7].w[i]);
        }
    };
    BinItem<W> v[SS_ITEMS];
    if (on) {
        uint32_t row[SS_ITEMS];
#pragma unroll
        for (int e = 0; e < SS_ITEMS; ++e) {
            const int i = warp * SS_WARP_ROWS + 32 * e + lane;
            row[e] = i < m ? (ids ? ids[i] : (uint32_t)i) : SS_NONE;
        }
#pragma unroll
        for (int e = 0; e < SS_ITEMS; ++e) {
            v[e].w[0] = row[e];
            if constexpr (W > 0) {
                uint4 k = make_uint4(0, 0, 0, 0);
                if (row[e] != SS_NONE) {
                    if constexpr (NW == 4) {
                        k = reinterpret_cast<const uint4*>(table)[row[e]];
                    } else {
                        const uint2 x = reinterpret_cast<const uint2*>(table)[row[e]];
                        k.z = x.x;
                        k.w = x.y;
                    }
                }
                uint32_t d[4];
                asm("sub.cc.u32 %0, %4, %8;\n\tsubc.cc.u32 %1, %5, %9;\n\tsubc.cc.u32 %2, %6, %10;\n\tsubc.u32 %3, %7, %11;"
                    : "=&r"(d[0]), "=&r"(d[1]), "=&r"(d[2]), "=&r"(d[3])
                    : "r"(k.w), "r"(k.z), "r"(k.y), "r"(k.x), "r"(low[3]), "r"(low[2]), "r"(low[1]), "r"(low[0]));
#pragma unroll
                for (int i = W - 1; i >= 0; --i) v[e].w[i + 1] = row[e] == SS_NONE ? 0xFFFFFFFFu : __funnelshift_l(i > 0 ? d[i - 1] : 0u, d[i], shift);
            }
        }
        warp_sort_items<W>(v, lane);
        store(v);
    }
    __syncthreads();
    // From a run of each warp: a thread finds by a search along its diagonal where its places of the merged run begin in the two.
    for (int run = SS_WARP_ROWS; run < padded; run *= 2) {
        if (on) {
            auto item = [&](int x) {
                BinItem<W> r;
#pragma unroll
                for (int i = 0; i <= W; ++i) r.w[i] = s_w[i][x];
                return r;
            };
            const int base = at & ~(2 * run - 1);
            const int ea = min(base + run, padded), eb = min(base + 2 * run, padded);
            const int d = at - base;
            int lo = max(0, d - (eb - ea)), hi = min(d, ea - base);
            while (lo < hi) {
                const int mid = (lo + hi) >> 1;
                const int x = ea + d - 1 - mid, y = base + mid;
                const uint32_t p = s_w[W][x], q = s_w[W][y];  // seldom the same
                if (p == q ? item_less<W>(item(x), item(y)) : p < q) hi = mid;
                else lo = mid + 1;
            }
            int ia = base + lo, ib = ea + d - lo;
            BinItem<W> a = item(min(ia, padded - 1)), b = item(min(ib, padded - 1));
#pragma unroll
            for (int e = 0; e < SS_ITEMS; ++e) {
                const bool first = ia < ea && (ib >= eb || !item_less<W>(b, a));
#pragma unroll
                for (int i = 0; i <= W; ++i) v[e].w[i] = first ? a.w[i] : b.w[i];
                const int next = first ? ++ia : ++ib;
                const BinItem<W> x = item(min(next, padded - 1));
#pragma unroll
                for (int i = 0; i <= W; ++i) {
                    a.w[i] = first ? x.w[i] : a.w[i];
                    b.w[i] = first ? b.w[i] : x.w[i];
                }
            }
        }
        __syncthreads();
        if (on) store(v);
        __syncthreads();
    }
}

// As splitter_bin_kernel, for the bins of more than `above` rows and, unless THREADS is SS_THREADS, of CAP at most.
template <int NW, int THREADS>
__global__ void __launch_bounds__(THREADS, 768 / THREADS)
splitter_short_bin_kernel(const uint32_t* __restrict__ keys, int n, int bins, const uint32_t* __restrict__ bin_start, RowList<NW> splitters, int above,
                     uint32_t* ids,
                     uint32_t* __restrict__ keys_out, uint32_t* __restrict__ ids_out) {
    constexpr int CAP = THREADS * SS_ITEMS;
    __shared__ __align__(16) uint32_t s_w[NW + 1][CAP];
    const int tid = threadIdx.x;
    const int t = blockIdx.x / bins, b = blockIdx.x - t * bins;
    const uint32_t first = ids ? bin_start[(size_t)t * (bins + 1) + b] : 0u;
    const int m_all = ids ? (int)(bin_start[(size_t)t * (bins + 1) + b + 1] - first) : n;
    if (m_all <= above || (THREADS < SS_THREADS && m_all > CAP)) return;
    const uint32_t* table = keys + (size_t)t * n * NW;
    const size_t base = (size_t)t * n + first;
    // the keys of the bin are these at least, and no more than that apart
    uint32_t low[4] = {0, 0, 0, 0};
    int words = NW, shift = 0;
    if (ids) {
        uint64_t a[2] = {0, 0}, z[2] = {NW == 4 ? ~0ull : 0ull, ~0ull};
        const size_t at = (size_t)t * bins + b;
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            if (b > 0) a[i] = splitters.p[i][at - 1];
            if (b < bins - 1) z[i] = splitters.p[i][at];
            low[2 * i] = (uint32_t)(a[i] >> 32);
            low[2 * i + 1] = (uint32_t)a[i];
        }
        const uint64_t d1 = z[1] - a[1], d0 = z[0] - a[0] - (z[1] < a[1] ? 1u : 0u);
        words = d0 >> 32 ? 4 : d0 ? 3 : d1 >> 32 ? 2 : d1 ? 1 : 0;
        shift = words ? __clzll((long long)(d0 ? d0 : d1)) & 31 : 0;
    }
    auto go = [&](auto tag) {
        constexpr int W = decltype(tag)::value;
        for (int c0 = 0; c0 < m_all; c0 += CAP) {
            const int m = min(CAP, m_all - c0);
            if (c0) __syncthreads();  // the piece before is out
            sort_bin<NW, W, CAP>(table, ids ? ids + base + c0 : nullptr, m, low, shift, s_w);
            if (m_all > CAP) {  // a piece: its rows in order where they were
                for (int i = tid; i < m; i += THREADS) ids[base + c0 + i] = s_w[0][i];
                continue;
            }
            for (int i = tid; i < m; i += THREADS) {
                uint32_t d[5] = {0, 0, 0, 0, 0}, k[4];
#pragma unroll
                for (int j = 0; j < W; ++j) d[j] = s_w[j + 1][i];
#pragma unroll
                for (int j = 0; j < W; ++j) d[j] = __funnelshift_r(d[j], d[j + 1], shift);
                asm("add.cc.u32 %0, %4, %8;\n\taddc.cc.u32 %1, %5, %9;\n\taddc.cc.u32 %2, %6, %10;\n\taddc.u32 %3, %7, %11;"
                    : "=&r"(k[0]), "=&r"(k[1]), "=&r"(k[2]), "=&r"(k[3])
                    : "r"(d[0]), "r"(d[1]), "r"(d[2]), "r"(d[3]), "r"(low[3]), "r"(low[2]), "r"(low[1]), "r"(low[0]));
                if constexpr (NW == 4) reinterpret_cast<uint4*>(keys_out)[base + i] = make_uint4(k[3], k[2], k[1], k[0]);
                else reinterpret_cast<uint2*>(keys_out)[base + i] = make_uint2(k[1], k[0]);
                ids_out[base + i] = s_w[0][i];
            }
        }
    };
    if constexpr (NW == 4) {
        if (words == 4) go(std::integral_constant<int, 4>{});
        else if (words == 3) go(std::integral_constant<int, 3>{});
    }
    if (words == 2) go(std::integral_constant<int, 2>{});
    else if (words == 1) go(std::integral_constant<int, 1>{});
    else if (words == 0) go(std::integral_constant<int, 0>{});
    if (THREADS == SS_THREADS && m_all > CAP) place_pieces<NW>(table, 0, ids + base, m_all, keys_out + base * NW, ids_out + base);
}

// ---------------------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------------------
struct SplitterPlan {
    int bins, samples, chunks, tile, tiles;
    size_t hist, total, start, list, sorted, words;  // offsets into the scratch, in words
};
inline SplitterPlan splitter_plan(int n, int L) {
    SplitterPlan p{};
    p.bins = splitter_bins(n);
    p.samples = std::max(512, p.bins * SS_OVER);  // powers of two
    p.chunks = (int)ceil_div(p.samples, SS_CAP);
    // Short tiles fill the chip, but have as many counts as there are bins each: eight rows a bin at least (4 tables of 4M keys of 8 bytes, the sort with
    // tiles of 4,096 1,570 us, of 16,384 1,115; one table of 100,003 97 and 106, of 1M 165, with 8,192 160, and 176).
    p.tile = (size_t)L * ceil_div(n, SS_TILE) < 1024 ? std::min(std::max(SS_SHORT_TILE, 8 * p.bins), SS_TILE) : SS_TILE;
    p.tiles = (int)ceil_div(n, p.tile);
    constexpr size_t row_words = 5;  // of a RowList
    auto take = [&](size_t words) {
        const size_t at = p.words;
        p.words += (words + 3) / 4 * 4;
        return at;
    };
    if (p.bins > 1) {
        p.hist = take((size_t)L * p.tiles * p.bins);
        p.total = take((size_t)L * p.bins);
        p.start = take((size_t)L * (p.bins + 1));
        p.list = take((size_t)L * p.bins * row_words);
        if (p.chunks > 1) p.sorted = take((size_t)L * p.samples * row_words);
    }
    return p;
}
// Keys this sort takes: of two words and more, in tables of up to 2^22 rows.  (8 tables of 16-byte keys, by radix passes and this way: 2^22 rows 3,712
// and 2,535 us, one more 3,737 by radix passes.)
inline bool splitters_can(int n, int NW) { return NW >= 2 && splitter_bins(n) <= SS_MAX_BINS; }

// What sorts the tables: splitters, or the radix sorts.  What a radix sort costs grows with the bytes of a key, what this costs with the logarithm
// of the rows; up to SS_CAP rows a table is one bin.  Above, this pays for keys of seven bytes and more that are not sorted in compressed form.  The sort stage by
// radix passes and this way: 32 tables of 16-byte keys, 1,000 rows 53 and 22 us, 30,000 316 and 132, 100,003 570 and 265, 500,000 1,789 and 1,051, 2M
// 6,061 and 4,134; 5-byte keys, 16 tables of 1M 741 and 826.
// CULSH_SORT_SPLITTERS=0 / 1: never / wherever it can.
//
// Rows of a table that the radix sort takes in one launch (one CTA or a cluster) and sorts faster or as fast.  It gains where keys repeat, and the more so
// the fewer bytes they have.  8 tables, all keys different, twenty rows to a key, ten keys in all: 12,289 rows of 16 bytes 95 and 69 us, 74 and 77, 68 and 85;
// 16,385 of 12 bytes in 0.71, 1.20 and 1.22 of the radix sort's time; 24,576 of 10 bytes 0.92, 1.26 and 1.48, 40,000 0.74, 1.05 and 1.20; of 11 bytes
// 0.81, 1.19 and 1.42, 0.65, 0.96 and 1.17; of 9 bytes 1.07, 1.37 and 1.62, 0.83, 1.12 and 1.39, of 8 and 7 alike.
inline int64_t splitters_from(int KB) { return KB >= 13 ? 12288 : KB == 12 ? 16384 : KB >= 10 ? 32768 : INT32_MAX; }
// Rows of a table up to which this is faster than radix passes with launches of their own, or as fast.  They gain with the rows, most of all beyond 2^21, where
// 4,096 splitters leave an SM no second CTA of the search, and with fewer tables.  Times by radix passes and this way:
//   7 bytes (this way with the 17 us of a look for a compressed form): 8 tables of 100,003 136 and 116 us, 131,072 138 and 143, 250,000 181 and 180, 1M 416
//   and 475, 2^22 1,516 and 2,249
//   8 bytes: 4 tables of 500,000 191 and 187 (twenty rows to a key 180 and 189), 786,432 with twenty rows to a key 213 and 240, 2^21 509 and 543, 2^22 966
//   and 1,140; 8 of 1M 483 and 460, 2^21 964 and 908, 3M 1,333 and 1,577
//   9 bytes: 4 of 1M 335 and 326, 2^21 569 and 597; 8 of 2^21 1,050 and 982, 3M 1,548 and 1,753; 10 bytes: 2 of 1M 246 and 234, 2^21 358 and 369; 8 of 2^21
//   1,130 and 1,018, 3M 1,662 and 1,733
//   11 bytes: 2 of 2^21 384 and 363, 3M 527 and 556; 8 of 3M 1,784 and 1,746, 2^22 2,568 and 2,398; 12 bytes: one of 3M 348 and 359
inline int64_t splitters_to(int KB, int L) {
    switch (KB) {
        case 7: return 7 << 14;
        case 8: return L < 8 ? 1 << 19 : 1 << 21;
        case 9: return L < 8 ? 1 << 20 : 1 << 21;
        case 10: return L < 4 ? 1 << 20 : 1 << 21;
        case 11: return L < 4 ? 1 << 21 : 1 << 22;
        default: return KB < 7 ? 0 : 1 << 22;
    }
}
inline bool sort_by_splitters(const CtxPtr& c, int n, int L, int NW, int KB, bool compressed) {
    if (!splitters_can(n, NW)) return false;
    const char* e = getenv("CULSH_SORT_SPLITTERS");
    if (e && *e) return atoi(e) != 0;
    if (n <= SS_CAP) return true;
    if (compressed || n > splitters_to(KB, L)) return false;
    return n > splitters_from(KB) || !radix_sort_is_small(c, n, L, NW, compressed);
}

// keys[0] -> keys[1], row ids to vals[1]; vals[0] is scratch.
template <int NW>
inline int splitter_sort_tables(const CtxPtr& c, uint32_t* keys[2], uint32_t* vals[2], int n, int L, int KB, uint32_t* scratch) {
    cudaStream_t s = c->stream;
    const SplitterPlan p = splitter_plan(n, L);
    const int skip = NW > 4 ? std::min(NW - 4, NW - (int)ceil_div(KB, 4)) : 0;
    auto list = [&](size_t at, size_t rows) {
        RowList<NW> r{};
        r.p[0] = reinterpret_cast<uint64_t*>(scratch + at);
        r.p[1] = r.p[0] + rows;
        r.id = reinterpret_cast<uint32_t*>(r.p[1] + rows);
        return r;
    };
    auto smem_of = [&](auto kern, size_t smem) { CU_CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem)); };
    constexpr size_t sort_smem = sizeof(typename BlockSort<NW>::Smem);
    uint32_t* ids = nullptr;
    if (p.bins > 1) {
        const RowList<NW> splitters = list(p.list, (size_t)L * p.bins), sorted = p.chunks > 1 ? list(p.sorted, (size_t)L * p.samples) : splitters;
        auto sample = splitter_sample_kernel<NW>;
        smem_of(sample, sort_smem);
        launch_next(s, sample, (unsigned)(L * p.chunks), SS_THREADS, sort_smem, keys[0], n, skip, p.samples, p.chunks, p.bins,
                    p.samples / p.bins, sorted);
        KERNEL_CHECK();
        if (p.chunks > 1) {
            const int total = L * p.samples;
            launch_next(s, splitter_rank_kernel<NW>, (unsigned)ceil_div(total, 256), 256, 0, keys[0], n, skip, p.chunks, p.bins, total, sorted, splitters);
            KERNEL_CHECK();
        }
        uint16_t* bin_of = reinterpret_cast<uint16_t*>(keys[1]);  // until the keys come
        auto classify = splitter_classify_kernel<NW>;
        smem_of(classify, splitter_classify_smem(p.bins));
        classify<<<(unsigned)(L * p.tiles), SS_TILE_THREADS, splitter_classify_smem(p.bins), s>>>(keys[0], n, skip, p.tile, p.tiles, p.bins, splitters,
                                                                                                bin_of, scratch + p.hist);
        KERNEL_CHECK();
        launch_next(s, splitter_scan_kernel, (unsigned)ceil_div((size_t)L * p.bins, SS_SCAN_THREADS), SS_SCAN_THREADS, 0, scratch + p.hist, p.tiles, p.bins,
                                                                                                           L * p.bins, scratch + p.total);
        KERNEL_CHECK();
        ids = vals[0];
        smem_of(splitter_scatter_kernel, splitter_scatter_smem(p.tile, p.bins));
        launch_next(s, splitter_scatter_kernel, (unsigned)(L * p.tiles), SS_TILE_THREADS, splitter_scatter_smem(p.tile, p.bins),
            bin_of, n, p.tile, p.tiles, p.bins, scratch + p.hist, scratch + p.total, scratch + p.start, ids);
        KERNEL_CHECK();
    }
    if (c->profiling) cudaEventRecord(c->ev_pass[0], s);
    if constexpr (NW <= 4) {
        // half the bins need half a CTA, and a CTA of that size leaves no registers idle
        const RowList<NW> splitters = list(p.list, (size_t)L * p.bins);
        constexpr int HALF = SS_THREADS / 2;
        const bool halves = p.bins > 1 || n <= HALF * SS_ITEMS, wholes = p.bins > 1 || !halves;
        if (halves) {
            splitter_short_bin_kernel<NW, HALF><<<(unsigned)(L * p.bins), HALF, 0, s>>>(keys[0], n, p.bins, scratch + p.start, splitters, -1, ids,
                                                                                     keys[1], vals[1]);
            KERNEL_CHECK();
        }
        if (wholes) {
            splitter_short_bin_kernel<NW, SS_THREADS><<<(unsigned)(L * p.bins), SS_THREADS, 0, s>>>(
                keys[0], n, p.bins, scratch + p.start, splitters, halves ? HALF * SS_ITEMS : -1, ids, keys[1], vals[1]);
            KERNEL_CHECK();
        }
    } else {
        auto bin = splitter_bin_kernel<NW>;
        smem_of(bin, sort_smem);
        bin<<<(unsigned)(L * p.bins), SS_THREADS, sort_smem, s>>>(keys[0], n, skip, p.bins, scratch + p.start, ids, keys[1], vals[1]);
        KERNEL_CHECK();
    }
    if (c->profiling) cudaEventRecord(c->ev_pass[1], s);
    return 1;
}

}  // namespace culsh_b200
