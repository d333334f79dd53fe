// Per-table stable LSD radix sort of (packed key, row id) pairs, all tables in one launch
// per 8-bit digit.  Replaces upstream's loop of extract_byte_key_kernel +
// cub::DeviceRadixSort::SortPairs per signature byte plus the table-id pass
// (core/fit.cuh:254-282): here the packed key travels with the row id, so no pass gathers
// signature bytes at random, and tables never mix (a tile belongs to one table).  A pass is
// three launches - tile histograms, a per-table scan that turns them into destination
// offsets, and the stable scatter - so no CTA ever waits on another one: a chained
// look-back between tiles was measured to cost more than the extra 4 bytes per item that
// the histogram read adds at this bandwidth.
//
// P-stable keys of one byte per hash (at most eight hashes) whose values span at most 32 levels
// are sorted in COMPRESSED form: the first pass replaces every key byte by its 5-bit rank among
// the values in use and packs the ranks (hash 0 most significant), the passes in between see a
// key of 5 bits per hash - 5 passes instead of 8 for eight hashes -, and the last pass writes the
// original bytes back.  The rank keeps the unsigned order of the byte (non-negative values
// first, then the negative ones, two's complement bytes 128..255), so the sorted order is the
// one a byte-per-pass sort of the original keys gives.  When such a key takes two words (five to
// eight hashes: at most 40 bits compressed) and the table has at most 2^24 rows, the compressed
// key and the row id travel PACKED in one 64-bit item (key << 24 | id) between the first and the
// last pass: 8 bytes per item instead of 12 and no separate id array in the passes in between.
//
// Keys of four words and more (MinHash from three hashes on, wide p-stable keys), in tables too long for the splitters
// (see splitter_sort.cuh, which takes most of them), stay where they are: the
// sort runs over one word of the key at a time, least significant first, and what it moves are
// (word, row id) pairs.  See radix_sort_words.
#pragma once

#include <type_traits>

#include "common.cuh"
#include "index_math.h"

namespace culsh_b200 {

constexpr int RS_THREADS = 256;
constexpr int RS_WARPS = RS_THREADS / 32;

template <int NW>
struct SortCfg {
    // items per thread: as many as leave a tile's keys in registers at four CTAs per SM
    static constexpr int IPT = NW == 1 ? 16 : 12;
    static constexpr int TILE = RS_THREADS * IPT;
    static constexpr size_t SMEM =
        sizeof(uint32_t) * ((size_t)TILE * NW + TILE + RS_WARPS * 256 + 256 + 32);
};

inline int sort_tile_items(int NW) { return NW == 2 ? SortCfg<2>::TILE : SortCfg<1>::TILE; }

template <int NW>
__device__ __forceinline__ void load_key(const uint32_t* __restrict__ src, uint32_t* k) {
    if (NW == 1) {
        k[0] = src[0];
    } else if (NW == 2) {
        uint2 v = *reinterpret_cast<const uint2*>(src);
        k[0] = v.x; k[1] = v.y;
    } else {
#pragma unroll
        for (int i = 0; i < NW / 4; ++i) {
            uint4 v = reinterpret_cast<const uint4*>(src)[i];
            k[4 * i] = v.x; k[4 * i + 1] = v.y; k[4 * i + 2] = v.z; k[4 * i + 3] = v.w;
        }
    }
}

template <int NW>
__device__ __forceinline__ void store_key(uint32_t* __restrict__ dst, const uint32_t* k) {
    if (NW == 1) {
        dst[0] = k[0];
    } else if (NW == 2) {
        *reinterpret_cast<uint2*>(dst) = make_uint2(k[0], k[1]);
    } else {
#pragma unroll
        for (int i = 0; i < NW / 4; ++i)
            reinterpret_cast<uint4*>(dst)[i] =
                make_uint4(k[4 * i], k[4 * i + 1], k[4 * i + 2], k[4 * i + 3]);
    }
}

// ---------------------------------------------------------------------------------------
// Compressed form of one-byte-per-hash keys (NW = 1 or 2).  rank(u) = u for a byte below 128
// (n_pos such values in use: 0 .. n_pos-1), u - sub for a byte from 128 up, with
// sub = smallest negative byte - n_pos; every rank is below 32.
// ---------------------------------------------------------------------------------------
struct KeyComp {
    uint32_t sub;    // see above
    uint32_t n_pos;  // ranks below n_pos are non-negative values
};

// From the self-check word and the range behind it (see HashRange): whether the values span at most 32 levels.
__host__ __device__ inline bool key_comp_of(int err, int lo, int hi, KeyComp& kc) {
    const uint32_t n_pos = (uint32_t)hi + 1, n_neg = (uint32_t)-lo;
    if (err || n_pos + n_neg > 32) return false;
    kc.n_pos = n_pos;
    kc.sub = n_neg ? 256u - n_neg - n_pos : 0u;
    return true;
}

__device__ __forceinline__ uint32_t comp_word(uint32_t w, uint32_t sub) {  // 4 bytes -> 20 bits
    const uint32_t neg = (w >> 7) & 0x01010101u;
    uint32_t c = w - neg * sub;                                   // four ranks, one per byte
    c = (c & 0x001F001Fu) | ((c & 0x1F001F00u) >> 3);             // two 10-bit fields
    return (c & 0x3FFu) | ((c >> 6) & 0xFFC00u);
}
__device__ __forceinline__ uint32_t decomp_word(uint32_t c20, KeyComp kc) {  // 20 bits -> 4 bytes
    uint32_t c = (c20 & 0x3FFu) | ((c20 & 0xFFC00u) << 6);
    c = (c & 0x001F001Fu) | ((c << 3) & 0x1F001F00u);
    uint32_t w = 0;
#pragma unroll
    for (int b = 0; b < 4; ++b) {
        const uint32_t r = (c >> (8 * b)) & 0xFFu;
        w |= (r + (r >= kc.n_pos ? kc.sub : 0u)) << (8 * b);
    }
    return w;
}
template <int NW>
__device__ __forceinline__ void comp_key(uint32_t* k, uint32_t sub) {
    if (NW == 1) {
        k[0] = comp_word(k[0], sub);
    } else {
        const uint64_t v = ((uint64_t)comp_word(k[0], sub) << 20) | comp_word(k[1], sub);
        k[0] = (uint32_t)(v >> 32);
        k[1] = (uint32_t)v;
    }
}
template <int NW>
__device__ __forceinline__ void decomp_key(uint32_t* k, KeyComp kc) {
    if (NW == 1) {
        k[0] = decomp_word(k[0], kc);
    } else {
        const uint64_t v = ((uint64_t)k[0] << 32) | k[1];
        k[0] = decomp_word((uint32_t)(v >> 20) & 0xFFFFFu, kc);
        k[1] = decomp_word((uint32_t)v & 0xFFFFFu, kc);
    }
}

// ---------------------------------------------------------------------------------------
// Pass step 1: digit histogram of every tile (a tile is TILE consecutive items of one
// table).  tile_hist layout: [tile][256].
// ---------------------------------------------------------------------------------------
template <int NW, bool COMP0>
__global__ void __launch_bounds__(RS_THREADS)
radix_tile_hist_kernel(const uint32_t* __restrict__ keys, int n, int tiles_per_table, int p, uint32_t sub,
                       uint32_t* __restrict__ tile_hist, KernelBefore kernel_before) {
    behind_kernel_before(keys, tile_hist, kernel_before);
    using Cfg = SortCfg<NW>;
    __shared__ uint32_t s_hist[256];
    const int tile = blockIdx.x;
    const int t = tile / tiles_per_table;
    const int lt = tile - t * tiles_per_table;
    const int item0 = lt * Cfg::TILE;
    const int count = min(Cfg::TILE, n - item0);
    const uint32_t* base = keys + ((size_t)t * n + item0) * NW + (NW - 1 - (p >> 2));
    const int shift = 8 * (p & 3);
    s_hist[threadIdx.x] = 0;
    __syncthreads();
    if (COMP0) {  // p == 0 of a compressed sort: the digit is the low byte of the compressed key
        const uint32_t* last = keys + ((size_t)t * n + item0) * NW + (NW - 1);
#pragma unroll 4
        for (int i = threadIdx.x; i < count; i += RS_THREADS)
            atomicAdd(&s_hist[comp_word(last[(size_t)i * NW], sub) & 0xFFu], 1u);
    } else {
#pragma unroll 4
        for (int i = threadIdx.x; i < count; i += RS_THREADS)
            atomicAdd(&s_hist[(base[(size_t)i * NW] >> shift) & 0xFFu], 1u);
    }
    __syncthreads();
    tile_hist[(size_t)tile * 256 + threadIdx.x] = s_hist[threadIdx.x];
}

// ---------------------------------------------------------------------------------------
// Pass step 2: one block per table turns the tile histograms into the offset (inside the
// table) at which each tile's run of each digit starts:
//   off[tile][d] = sum over d' < d of total[d'] + sum over earlier tiles of hist[tile'][d].
// 1024 threads = 4 tile segments x 256 digits.
// ---------------------------------------------------------------------------------------
constexpr int RS_SCAN_THREADS = 1024;
constexpr int RS_SCAN_SEGS = RS_SCAN_THREADS / 256;

__global__ void __launch_bounds__(RS_SCAN_THREADS)
radix_tile_scan_kernel(uint32_t* __restrict__ tile_hist, int tiles_per_table, KernelBefore kernel_before) {
    behind_kernel_before(tile_hist, kernel_before);
    __shared__ uint32_t s_seg[RS_SCAN_SEGS][256];
    __shared__ uint32_t s_base[256];
    __shared__ uint32_t s_warp[8];
    const int d = threadIdx.x & 255, seg = threadIdx.x >> 8;
    uint32_t* h = tile_hist + (size_t)blockIdx.x * tiles_per_table * 256 + d;
    const int per_seg = (tiles_per_table + RS_SCAN_SEGS - 1) / RS_SCAN_SEGS;
    const int i0 = seg * per_seg, i1 = min(tiles_per_table, i0 + per_seg);
    uint32_t sum = 0;
#pragma unroll 8
    for (int i = i0; i < i1; ++i) sum += h[(size_t)i * 256];
    s_seg[seg][d] = sum;
    __syncthreads();
    if (seg == 0) {  // exclusive scan of the digit totals over the 256 digits
        uint32_t tot = 0;
#pragma unroll
        for (int g = 0; g < RS_SCAN_SEGS; ++g) tot += s_seg[g][d];
        const int lane = d & 31, w = d >> 5;
        uint32_t inc = tot;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            uint32_t x = __shfl_up_sync(0xFFFFFFFFu, inc, o);
            if (lane >= o) inc += x;
        }
        if (lane == 31) s_warp[w] = inc;
        s_base[d] = inc - tot;  // exclusive inside the warp; the warp bases are added below
    }
    __syncthreads();
    uint32_t run = s_base[d];
    for (int w = 0; w < (d >> 5); ++w) run += s_warp[w];
    for (int g = 0; g < seg; ++g) run += s_seg[g][d];
#pragma unroll 8
    for (int i = i0; i < i1; ++i) {
        uint32_t x = h[(size_t)i * 256];
        h[(size_t)i * 256] = run;
        run += x;
    }
}

// Tables with many tiles: one block per (table, chunk of RS_CHUNK_TILES tiles) scans its chunk
// on its own (exclusive prefix over the chunk's tiles per digit, chunk totals on the side), a
// second tiny launch turns the chunk totals into chunk bases (digit prefix + earlier chunks), and
// the scatter adds the base of its chunk.  With one block per table the scan of a 10M-row table
// (2441 tiles) ran on 48 SMs for 1.2 ms per pass; at 244 tiles x 32 tables a scan takes 7 us in chunks of
// 64 tiles and 2 more for the bases, in place of 15 by one block per table.
constexpr int RS_CHUNK_TILES = 64;
constexpr int RS_CHUNK_MIN_TILES = 96;  // tables with fewer tiles keep the single-launch scan

__global__ void __launch_bounds__(RS_SCAN_THREADS)
radix_tile_scan_chunk_kernel(uint32_t* __restrict__ tile_hist, int tiles_per_table, int n_chunks,
                             uint32_t* __restrict__ chunk_tot /* [table][chunk][256] */, KernelBefore kernel_before) {
    behind_kernel_before(tile_hist, chunk_tot, kernel_before);
    __shared__ uint32_t s_seg[RS_SCAN_SEGS][256];
    const int d = threadIdx.x & 255, seg = threadIdx.x >> 8;
    const int table = blockIdx.x / n_chunks, chunk = blockIdx.x - table * n_chunks;
    const int t_begin = chunk * RS_CHUNK_TILES, t_end = min(tiles_per_table, t_begin + RS_CHUNK_TILES);
    uint32_t* h = tile_hist + (size_t)table * tiles_per_table * 256 + d;
    const int per_seg = (t_end - t_begin + RS_SCAN_SEGS - 1) / RS_SCAN_SEGS;
    const int i0 = t_begin + seg * per_seg, i1 = min(t_end, i0 + per_seg);
    uint32_t sum = 0;
#pragma unroll 8
    for (int i = i0; i < i1; ++i) sum += h[(size_t)i * 256];
    s_seg[seg][d] = sum;
    __syncthreads();
    uint32_t run = 0, tot = 0;
#pragma unroll
    for (int g = 0; g < RS_SCAN_SEGS; ++g) {
        const uint32_t x = s_seg[g][d];
        if (g < seg) run += x;
        tot += x;
    }
    if (seg == 0) chunk_tot[(size_t)blockIdx.x * 256 + d] = tot;
#pragma unroll 8
    for (int i = i0; i < i1; ++i) {
        const uint32_t x = h[(size_t)i * 256];
        h[(size_t)i * 256] = run;
        run += x;
    }
}

// one block of 256 threads per table: chunk_tot -> chunk bases, in place
__global__ void __launch_bounds__(256)
radix_chunk_base_kernel(uint32_t* __restrict__ chunk_tot, int n_chunks, KernelBefore kernel_before) {
    behind_kernel_before(chunk_tot, kernel_before);
    __shared__ uint32_t s_warp[8];
    const int d = threadIdx.x, lane = d & 31, w = d >> 5;
    uint32_t* ct = chunk_tot + (size_t)blockIdx.x * n_chunks * 256 + d;
    uint32_t tot = 0;
    for (int c = 0; c < n_chunks; ++c) tot += ct[(size_t)c * 256];
    uint32_t inc = tot;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t x = __shfl_up_sync(0xFFFFFFFFu, inc, o);
        if (lane >= o) inc += x;
    }
    if (lane == 31) s_warp[w] = inc;
    __syncthreads();
    uint32_t run = inc - tot;
    for (int i = 0; i < w; ++i) run += s_warp[i];
    for (int c = 0; c < n_chunks; ++c) {
        const uint32_t x = ct[(size_t)c * 256];
        ct[(size_t)c * 256] = run;
        run += x;
    }
}

// ---------------------------------------------------------------------------------------
// Pass step 3: stable scatter of one tile on byte `p`.
//
// Shared memory and the latency between its phases bound it, not HBM (8-byte items move at 3.9 TB/s of
// the 6.5 a copy reaches).  Ranking costs a random shared-memory read and a write of the digits' last
// lanes per 32 items; counting with atomics and a broadcast of their result took a shuffle and a second random read
// in the reorder more, and words of lane bits set with atomicOr were slower where digits repeat.
// Whole tiles have no bounds in the code.  480M items of 4 + 4 bytes: 2.66 -> 2.0 ms a pass; 200M packed
// items of 8 bytes: first pass 1.59 -> 0.87, middle ones 1.26 -> 0.73, last 1.25 -> 0.90.
// ---------------------------------------------------------------------------------------
// Takes the lanes that differ from this one in the bit `mask` of d out of `lanes`: the step of CUB's MatchAny
// (cub/util_ptx.cuh: test, ballot, complement where the bit is clear, and).  Spelled out because the
// scatter is bound by what it issues: with a ballot and a select in C++ 32M items of 4 + 4 bytes took 155 us a
// pass, this way 128.
__device__ __forceinline__ void keep_same_bit(uint32_t& lanes, uint32_t d, uint32_t mask) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .b32 t, m;\n\t"
        "and.b32 t, %1, %2;\n\t"
        "setp.ne.b32 p, t, 0;\n\t"
        "vote.sync.ballot.b32 m, p, 0xffffffff;\n\t"
        "@!p not.b32 m, m;\n\t"
        "and.b32 %0, %0, m;\n\t}"
        : "+r"(lanes)
        : "r"(d), "r"(mask));
}

// COMP: 0 plain keys; 1 first pass of a compressed sort (keys are compressed as they are
// loaded); 2 its last pass (the original bytes are written back); 3 plain keys that nobody reads
// after this pass (the last one over a word of a wide key): only the ids are written.
// PACK (NW = 2, compressed): items are (compressed key << 24 | row id); the digit of pass p is
// byte p + 3 of the item, ids are neither loaded nor stored except by the last pass.
constexpr int RS_PACK_ID_BITS = 24;

template <int NW, bool FIRST, int COMP, bool PACK = false>
__global__ void __launch_bounds__(RS_THREADS, 4)
radix_scatter_kernel(const uint32_t* __restrict__ keys_in, const uint32_t* __restrict__ vals_in,
                     uint32_t* __restrict__ keys_out, uint32_t* __restrict__ vals_out, int n,
                     int tiles_per_table, int p, KeyComp kc, const uint32_t* __restrict__ tile_off,
                     const uint32_t* __restrict__ chunk_base /* or null */, int n_chunks, KernelBefore kernel_before) {
    behind_kernel_before(keys_in, vals_in, keys_out, vals_out, tile_off, chunk_base, kernel_before);
    using Cfg = SortCfg<NW>;
    constexpr int IPT = Cfg::IPT;
    constexpr int TILE = Cfg::TILE;
    extern __shared__ __align__(16) uint32_t smem[];
    uint32_t* s_keys = smem;                                            // [TILE][NW]
    uint32_t* s_vals = s_keys + (size_t)TILE * NW;                      // [TILE]
    uint32_t* s_bins = s_vals + TILE;                                   // [RS_WARPS][256] counts, then starts
    uint32_t* s_gdst = s_bins + RS_WARPS * 256;                         // [256] global dst of local position 0 of a bin
    uint32_t* s_misc = s_gdst + 256;                                    // [32]

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int tile = blockIdx.x;
    const int t = tile / tiles_per_table;
    const int lt = tile - t * tiles_per_table;
    const int item0 = lt * TILE;
    const int count = min(TILE, n - item0);
    const size_t base = (size_t)t * n + item0;
    const int pd = PACK ? p + 3 : p;  // byte of the item that holds this pass's digit
    const int dword = NW - 1 - (pd >> 2), dshift = 8 * (pd & 3);
    auto digit = [&](const uint32_t* key) {
        uint32_t word = key[0];
#pragma unroll
        for (int w = 1; w < NW; ++w)  // select chain keeps the key in registers
            if (w == dword) word = key[w];
        return (word >> dshift) & 0xFFu;
    };
    // needed late: fetched early, and summed only where used (an add here would stall the warp on
    // both loads before the key loads are issued)
    const uint32_t my_off = tile_off[(size_t)tile * 256 + tid];
    const uint32_t my_base = chunk_base ? chunk_base[((size_t)t * n_chunks + lt / RS_CHUNK_TILES) * 256 + tid] : 0u;
#pragma unroll
    for (int i = 0; i < RS_WARPS / 4; ++i) reinterpret_cast<uint4*>(s_bins)[i * RS_THREADS + tid] = make_uint4(0, 0, 0, 0);

    auto body = [&](auto full_tag) {
        constexpr bool FULL = decltype(full_tag)::value;  // whole tile: no bounds
        // ---- load (all loads in flight together) --------------------------------------
        uint32_t key[IPT][NW];
        uint32_t val[IPT];
        uint32_t pos[IPT];
        const int first = warp * (32 * IPT) + lane;
#pragma unroll
        for (int i = 0; i < IPT; ++i) {
            const int li = first + i * 32;
#pragma unroll
            for (int w = 0; w < NW; ++w) key[i][w] = 0;
            val[i] = 0;
            if (FULL || li < count) {
                load_key<NW>(keys_in + (base + li) * NW, key[i]);
                if constexpr (!PACK && !FIRST) val[i] = vals_in[base + li];
            }
        }
        if constexpr (COMP == 1) {
#pragma unroll
            for (int i = 0; i < IPT; ++i) {
                comp_key<NW>(key[i], kc.sub);
                if constexpr (PACK) {  // (40-bit compressed key) << 24 | row id
                    key[i][0] = (key[i][0] << RS_PACK_ID_BITS) | (key[i][NW - 1] >> (32 - RS_PACK_ID_BITS));
                    key[i][NW - 1] = (key[i][NW - 1] << RS_PACK_ID_BITS) | (uint32_t)(item0 + first + i * 32);
                }
            }
        }
        __syncthreads();
        // ---- rank inside the warp, 32 items a step: eight ballots give a lane the lanes that hold
        // its digit, every lane reads the digit's count of the steps before, and the highest lane of a digit
        // leaves the new one.  Lane order inside a digit keeps the sort stable. ----
        uint32_t* bins = s_bins + warp * 256;
        const uint32_t below = (1u << lane) - 1u;
#pragma unroll
        for (int i = 0; i < IPT; ++i) {
            const bool ok = FULL || first + i * 32 < count;
            const uint32_t d = digit(key[i]);
            uint32_t peers;
            if constexpr (COMP == 2) {
                peers = __match_any_sync(0xFFFFFFFFu, ok ? d : 0x100u);
            } else {
                peers = FULL ? 0xFFFFFFFFu : __ballot_sync(0xFFFFFFFFu, ok);
#pragma unroll
                for (int b = 0; b < 8; ++b) keep_same_bit(peers, d, 1u << b);
            }
            pos[i] = bins[d] + __popc(peers & below);
            __syncwarp();
            if (ok && (peers >> lane) == 1u) bins[d] = pos[i] + 1u;
            __syncwarp();
        }
        __syncthreads();

        // ---- per bin: tile count, start inside the tile, exclusive offsets of the warps ----
        uint32_t cnt = 0;
#pragma unroll
        for (int w = 0; w < RS_WARPS; ++w) cnt += s_bins[w * 256 + tid];
        uint32_t inc = cnt;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            uint32_t x = __shfl_up_sync(0xFFFFFFFFu, inc, o);
            if (lane >= o) inc += x;
        }
        if (lane == 31) s_misc[1 + warp] = inc;
        __syncthreads();
        uint32_t binstart = inc - cnt;
        for (int i = 0; i < warp; ++i) binstart += s_misc[1 + i];
        s_gdst[tid] = (uint32_t)((size_t)t * n) + my_off + my_base - binstart;
#pragma unroll
        for (int w = 0; w < RS_WARPS; ++w) {
            const uint32_t x = s_bins[w * 256 + tid];
            s_bins[w * 256 + tid] = binstart;
            binstart += x;
        }
        __syncthreads();

        // ---- reorder inside shared memory --------------------------------------------
#pragma unroll
        for (int i = 0; i < IPT; ++i) {
            if (FULL || first + i * 32 < count) {
                const uint32_t to = bins[digit(key[i])] + pos[i];
                store_key<NW>(s_keys + (size_t)to * NW, key[i]);
                if constexpr (!PACK) s_vals[to] = FIRST ? (uint32_t)(item0 + first + i * 32) : val[i];
            }
        }
        __syncthreads();

        // ---- coalesced runs out ------------------------------------------------------
#pragma unroll 4
        for (int i = 0; i < IPT; ++i) {
            const int at = i * RS_THREADS + tid;
            if (!FULL && at >= count) break;
            uint32_t kk[NW];
            load_key<NW>(s_keys + (size_t)at * NW, kk);
            const uint32_t g = s_gdst[digit(kk)] + (uint32_t)at;
            if constexpr (PACK) {
                if (COMP == 2) {  // unpack: id from the low bits, the key back to its two-word compressed form
                    vals_out[g] = kk[NW - 1] & ((1u << RS_PACK_ID_BITS) - 1u);
                    kk[NW - 1] = (kk[0] << (32 - RS_PACK_ID_BITS)) | (kk[NW - 1] >> RS_PACK_ID_BITS);
                    kk[0] >>= RS_PACK_ID_BITS;
                    decomp_key<NW>(kk, kc);
                }
                store_key<NW>(keys_out + (size_t)g * NW, kk);
            } else {
                if (COMP == 2) decomp_key<NW>(kk, kc);
                if (COMP != 3) store_key<NW>(keys_out + (size_t)g * NW, kk);
                vals_out[g] = s_vals[at];
            }
        }
    };
    if (count == TILE) body(std::true_type{});
    else body(std::false_type{});
}

// ---------------------------------------------------------------------------------------
// Wide keys: word `word` of the key of every item in the order reached so far (vals, or row order when
// it is null), and the tile histograms of its low byte on the way.
// ---------------------------------------------------------------------------------------
template <int NW>
__global__ void __launch_bounds__(RS_THREADS)
radix_word_gather_kernel(const uint32_t* __restrict__ keys, const uint32_t* __restrict__ vals, int n,
                         int tiles_per_table, int word, uint32_t* __restrict__ words, uint32_t* __restrict__ tile_hist) {
    using Cfg = SortCfg<1>;
    __shared__ uint32_t s_hist[256];
    const int tile = blockIdx.x;
    const int t = tile / tiles_per_table;
    const int item0 = (tile - t * tiles_per_table) * Cfg::TILE;
    const int count = min(Cfg::TILE, n - item0);
    const size_t base = (size_t)t * n + item0;
    const uint32_t* table = keys + (size_t)t * n * NW + word;
    s_hist[threadIdx.x] = 0;
    __syncthreads();
#pragma unroll 8
    for (int i = threadIdx.x; i < count; i += RS_THREADS) {
        const uint32_t id = vals ? vals[base + i] : (uint32_t)(item0 + i);
        const uint32_t w = table[(size_t)id * NW];
        words[base + i] = w;
        atomicAdd(&s_hist[w & 0xFFu], 1u);
    }
    __syncthreads();
    tile_hist[(size_t)tile * 256 + threadIdx.x] = s_hist[threadIdx.x];
}

// Keys in sorted order.
template <int NW>
__global__ void __launch_bounds__(RS_THREADS)
radix_key_gather_kernel(const uint32_t* __restrict__ keys, const uint32_t* __restrict__ vals, int n, int tiles_per_table,
                        uint32_t* __restrict__ out) {
    constexpr int Q = NW / 4;  // 16-byte quarters of a key, one per thread
    const int t = blockIdx.x / tiles_per_table;
    const size_t base = (size_t)t * n;
    const int64_t q0 = tile_first(blockIdx.x - t * tiles_per_table, RS_THREADS * 8);
    const uint4* src = reinterpret_cast<const uint4*>(keys) + base * Q;
    uint4* dst = reinterpret_cast<uint4*>(out) + base * Q;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int64_t q = q0 + i * RS_THREADS + threadIdx.x;
        if (q < (int64_t)n * Q) dst[q] = src[(size_t)vals[base + q / Q] * Q + q % Q];
    }
}

// ---------------------------------------------------------------------------------------
// Short tables: one CTA sorts a whole table, every pass in shared memory.  A pass of the general form is
// three launches, of which a table of a few thousand rows fills a few CTAs for 2 us each: what such a
// sort costs are its 15 launches (48 and more for keys of four words) and the gaps between them.
// 1,000 rows x 8 tables, five passes of packed items: 70 us of launches and gaps against 14 here; 10,000 x 16: 80
// against 40.  At the line it is still the faster one for every key and number of tables: 12,288 rows, one table, two
// byte passes 42 and 27, 64 passes of sixteen-word keys 1,101 and 602 (148 tables: 7,419 and 706).
// Above 12,288 items (8,192 of two words and an id) a table no longer fits the registers of one CTA.
// ---------------------------------------------------------------------------------------
constexpr int RSS_THREADS = 1024;
constexpr int RSS_WARPS = RSS_THREADS / 32;
template <int NW, bool PACK>
struct SmallSortCfg {
    static constexpr int KW = NW >= 4 ? 1 : NW;  // key words an item carries (wide keys: the word being sorted)
    static constexpr int IPT = KW == 1 || PACK ? 12 : 8;
    static constexpr int MAX_ROWS = RSS_THREADS * IPT;
    static constexpr size_t SMEM = sizeof(uint32_t) * ((size_t)MAX_ROWS * (KW + (PACK ? 0 : 1)) + RSS_WARPS * 256 + 4 * 256 + 256 + 8);
};

// COMP as a runtime flag: keys are compressed as they are loaded and restored as they are stored.  With
// `check` (the self-check word and the range) the kernel finds out itself whether they can be, which the host would have to
// wait for; where they cannot the items go through in row order, and the host, which sees that later, sorts again.
// Keys of eight and sixteen words are launched as usual: with pointers that the compiler knows nothing of their passes take 2.5 % longer.
template <int NW, bool PACK>
__global__ void __launch_bounds__(RSS_THREADS, 1)
radix_sort_small_kernel(const uint32_t* __restrict__ keys_in, uint32_t* __restrict__ keys_out,
                        uint32_t* __restrict__ vals_out, int n, int passes, bool compressed, KeyComp kc, const int* __restrict__ check, EarlyIf<(NW <= 4)> kernel_before) {
    behind_kernel_before(keys_in, keys_out, vals_out, check, kernel_before);
    using Cfg = SmallSortCfg<NW, PACK>;
    constexpr int KW = Cfg::KW, IPT = Cfg::IPT;
    constexpr bool WORDS = NW >= 4;
    extern __shared__ __align__(16) uint32_t smem[];
    uint32_t* s_keys = smem;                                     // [MAX_ROWS][KW]
    uint32_t* s_vals = s_keys + (size_t)Cfg::MAX_ROWS * KW;      // [MAX_ROWS], not packed
    uint32_t* s_bins = s_vals + (PACK ? 0 : Cfg::MAX_ROWS);      // [RSS_WARPS][256]
    uint32_t* s_part = s_bins + RSS_WARPS * 256;                 // [4][256]
    uint32_t* s_start = s_part + 4 * 256;                        // [256]
    uint32_t* s_warp = s_start + 256;                            // [8]

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const size_t base = (size_t)blockIdx.x * n;
    const int steps = (n + RSS_THREADS - 1) / RSS_THREADS;  // at most IPT
    const int first = warp * (32 * steps) + lane;           // a warp holds 32 * steps consecutive items
    const uint32_t below = (1u << lane) - 1u;
    uint32_t* bins = s_bins + warp * 256;
    if constexpr (!WORDS) {
        if (check && !key_comp_of(check[0], check[2], check[3], kc)) {
            for (int at = tid; at < n; at += RSS_THREADS) {
                uint32_t kk[KW];
                load_key<KW>(keys_in + (base + at) * KW, kk);
                store_key<KW>(keys_out + (base + at) * KW, kk);
                vals_out[base + at] = (uint32_t)at;
            }
            return;
        }
    }
    uint32_t key[IPT][KW], val[IPT], pos[IPT];
#pragma unroll
    for (int i = 0; i < IPT; ++i) {
        const int li = first + i * 32;
#pragma unroll
        for (int w = 0; w < KW; ++w) key[i][w] = 0;
        val[i] = (uint32_t)li;
        if (!WORDS && i < steps && li < n) {
            load_key<KW>(keys_in + (base + li) * KW, key[i]);
            if constexpr (!WORDS) {
                if (compressed) comp_key<KW>(key[i], kc.sub);
            }
            if constexpr (PACK) {
                key[i][0] = (key[i][0] << RS_PACK_ID_BITS) | (key[i][KW - 1] >> (32 - RS_PACK_ID_BITS));
                key[i][KW - 1] = (key[i][KW - 1] << RS_PACK_ID_BITS) | (uint32_t)li;
            }
        }
    }
    for (int p = 0; p < passes; ++p) {
        if (WORDS && (p & 3) == 0) {  // the next word of the key, from where the keys are
#pragma unroll
            for (int i = 0; i < IPT; ++i)
                if (i < steps && first + i * 32 < n) key[i][0] = keys_in[(base + val[i]) * NW + (NW - 1 - (p >> 2))];
        }
        const int pd = PACK ? p + 3 : (WORDS ? (p & 3) : p);
        const int dword = KW - 1 - (pd >> 2), dshift = 8 * (pd & 3);
        auto digit = [&](const uint32_t* k) { return ((KW == 2 && dword == 1 ? k[KW - 1] : k[0]) >> dshift) & 0xFFu; };
#pragma unroll
        for (int i = 0; i < RSS_WARPS * 256 / 4 / RSS_THREADS; ++i)
            reinterpret_cast<uint4*>(s_bins)[i * RSS_THREADS + tid] = make_uint4(0, 0, 0, 0);
        __syncthreads();
#pragma unroll
        for (int i = 0; i < IPT; ++i) {
            if (i < steps) {
                const bool ok = first + i * 32 < n;
                const uint32_t d = digit(key[i]);
                uint32_t peers = __ballot_sync(0xFFFFFFFFu, ok);
#pragma unroll
                for (int b = 0; b < 8; ++b) keep_same_bit(peers, d, 1u << b);
                pos[i] = bins[d] + __popc(peers & below);
                __syncwarp();
                if (ok && (peers >> lane) == 1u) bins[d] = pos[i] + 1u;
                __syncwarp();
            }
        }
        __syncthreads();
        // starts: a thread takes one bin and eight of the warps
        const int b = tid & 255, q = tid >> 8;
        uint32_t sum = 0;
#pragma unroll
        for (int w = 0; w < 8; ++w) sum += s_bins[(q * 8 + w) * 256 + b];
        s_part[tid] = sum;
        __syncthreads();
        if (tid < 256) {
            const uint32_t tot = s_part[tid] + s_part[256 + tid] + s_part[512 + tid] + s_part[768 + tid];
            uint32_t inc = tot;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t x = __shfl_up_sync(0xFFFFFFFFu, inc, o);
                if (lane >= o) inc += x;
            }
            if (lane == 31) s_warp[warp] = inc;
            s_start[tid] = inc - tot;
        }
        __syncthreads();
        uint32_t run = s_start[b];
        for (int w = 0; w < (b >> 5); ++w) run += s_warp[w];
        for (int g = 0; g < q; ++g) run += s_part[g * 256 + b];
#pragma unroll
        for (int w = 0; w < 8; ++w) {
            const uint32_t x = s_bins[(q * 8 + w) * 256 + b];
            s_bins[(q * 8 + w) * 256 + b] = run;
            run += x;
        }
        __syncthreads();
#pragma unroll
        for (int i = 0; i < IPT; ++i) {
            if (i < steps && first + i * 32 < n) {
                const uint32_t to = bins[digit(key[i])] + pos[i];
                store_key<KW>(s_keys + (size_t)to * KW, key[i]);
                if constexpr (!PACK) s_vals[to] = val[i];
            }
        }
        __syncthreads();
        if (p == passes - 1) break;
#pragma unroll
        for (int i = 0; i < IPT; ++i) {
            if (i < steps && first + i * 32 < n) {
                load_key<KW>(s_keys + (size_t)(first + i * 32) * KW, key[i]);
                if constexpr (!PACK) val[i] = s_vals[first + i * 32];
            }
        }
    }
    for (int at = tid; at < n; at += RSS_THREADS) {
        uint32_t id;
        if constexpr (WORDS) {
            id = s_vals[at];
            uint32_t kk[NW];
            load_key<NW>(keys_in + (base + id) * NW, kk);
            store_key<NW>(keys_out + (base + at) * NW, kk);
        } else {
            uint32_t kk[KW];
            load_key<KW>(s_keys + (size_t)at * KW, kk);
            if constexpr (PACK) {
                id = kk[KW - 1] & ((1u << RS_PACK_ID_BITS) - 1u);
                kk[KW - 1] = (kk[0] << (32 - RS_PACK_ID_BITS)) | (kk[KW - 1] >> RS_PACK_ID_BITS);
                kk[0] >>= RS_PACK_ID_BITS;
            } else {
                id = s_vals[at];
            }
            if (compressed) decomp_key<KW>(kk, kc);
            store_key<KW>(keys_out + (base + at) * KW, kk);
        }
        vals_out[base + at] = id;
    }
}

// ---------------------------------------------------------------------------------------
// The same with a cluster of CTAs for each table, while all tables' clusters find room at once: a CTA holds
// one stretch of the order, its digit totals go to all CTAs of the cluster, and an item is stored right into the shared
// memory of the CTA that holds its new place.  Two cluster barriers a pass keep the CTAs in step: totals are read after the first
// and items stored, which the second makes visible; what a barrier follows was read into registers before it.  What
// bounds it are the barriers and a warp's chain of steps.  Packed items, five passes: 10,000 rows x 16 tables with four CTAs 40 -> 25 us,
// 12,000 x 8 with eight 47 -> 21; 20,000 x 8, before in 15 launches, 81 -> 27, keys of four words in 49 289 -> 99.
// ---------------------------------------------------------------------------------------
constexpr int RSC_THREADS = 512;
constexpr int RSC_WARPS = RSC_THREADS / 32;
constexpr int RSC_MAX_CTAS = 8;  // the portable limit
template <int NW, bool PACK>
struct ClusterSortCfg {
    static constexpr int KW = SmallSortCfg<NW, PACK>::KW;
    static constexpr int IPT = SmallSortCfg<NW, PACK>::IPT;
    static constexpr int CTA_ROWS = RSC_THREADS * IPT;
    static constexpr size_t SMEM = sizeof(uint32_t) * ((size_t)CTA_ROWS * (KW + (PACK ? 0 : 1)) + RSC_WARPS * 256 + RSC_MAX_CTAS * 256 +
                                                       2 * 256 + 256 + 8);
};

template <int NW, bool PACK>
__global__ void __launch_bounds__(RSC_THREADS, 1)
radix_sort_cluster_kernel(const uint32_t* __restrict__ keys_in, uint32_t* __restrict__ keys_out,
                          uint32_t* __restrict__ vals_out, int n, int cta_rows, uint32_t cta_rows_inv, int passes, bool compressed,
                          KeyComp kc, const int* __restrict__ check, KernelBefore kernel_before) {
    behind_kernel_before(keys_in, keys_out, vals_out, check, kernel_before);
    using Cfg = ClusterSortCfg<NW, PACK>;
    constexpr int KW = Cfg::KW, IPT = Cfg::IPT;
    constexpr bool WORDS = NW >= 4;
    extern __shared__ __align__(16) uint32_t smem[];
    uint32_t* s_keys = smem;                                  // [CTA_ROWS][KW]
    uint32_t* s_vals = s_keys + (size_t)Cfg::CTA_ROWS * KW;   // [CTA_ROWS], not packed
    uint32_t* s_bins = s_vals + (PACK ? 0 : Cfg::CTA_ROWS);   // [RSC_WARPS][256]
    uint32_t* s_total = s_bins + RSC_WARPS * 256;             // [RSC_MAX_CTAS][256] of every CTA
    uint32_t* s_half = s_total + RSC_MAX_CTAS * 256;          // [2][256] of each half of the warps
    uint32_t* s_start = s_half + 2 * 256;                     // [256]
    uint32_t* s_warp = s_start + 256;                         // [8]

    auto cluster = cooperative_groups::this_cluster();
    const int ctas = (int)cluster.num_blocks(), rank = (int)cluster.block_rank();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int row0 = rank * cta_rows;  // place in the table
    const int count = max(0, min(cta_rows, n - row0));
    const size_t base = (size_t)(blockIdx.x / ctas) * n;
    const int steps = (cta_rows + RSC_THREADS - 1) / RSC_THREADS;  // at most IPT
    const int first = warp * (32 * steps) + lane;                 // a warp holds 32 * steps consecutive items
    const uint32_t below = (1u << lane) - 1u;
    uint32_t* bins = s_bins + warp * 256;
    if constexpr (!WORDS) {
        if (check && !key_comp_of(check[0], check[2], check[3], kc)) {  // every CTA of the cluster finds the same
            for (int at = tid; at < count; at += RSC_THREADS) {
                uint32_t kk[KW];
                load_key<KW>(keys_in + (base + row0 + at) * KW, kk);
                store_key<KW>(keys_out + (base + row0 + at) * KW, kk);
                vals_out[base + row0 + at] = (uint32_t)(row0 + at);
            }
            return;
        }
    }
    uint32_t key[IPT][KW], val[IPT], pos[IPT];
#pragma unroll
    for (int i = 0; i < IPT; ++i) {
        const int li = first + i * 32;
#pragma unroll
        for (int w = 0; w < KW; ++w) key[i][w] = 0;
        val[i] = (uint32_t)(row0 + li);
        if (!WORDS && i < steps && li < count) {
            load_key<KW>(keys_in + (base + row0 + li) * KW, key[i]);
            if constexpr (!WORDS) {
                if (compressed) comp_key<KW>(key[i], kc.sub);
            }
            if constexpr (PACK) {
                key[i][0] = (key[i][0] << RS_PACK_ID_BITS) | (key[i][KW - 1] >> (32 - RS_PACK_ID_BITS));
                key[i][KW - 1] = (key[i][KW - 1] << RS_PACK_ID_BITS) | (uint32_t)(row0 + li);
            }
        }
    }
    cluster.sync();  // all of them run: their shared memory may be written
    for (int p = 0; p < passes; ++p) {
        if (WORDS && (p & 3) == 0) {  // the next word of the key, from where the keys are
#pragma unroll
            for (int i = 0; i < IPT; ++i)
                if (i < steps && first + i * 32 < count) key[i][0] = keys_in[(base + val[i]) * NW + (NW - 1 - (p >> 2))];
        }
        const int pd = PACK ? p + 3 : (WORDS ? (p & 3) : p);
        const int dword = KW - 1 - (pd >> 2), dshift = 8 * (pd & 3);
        auto digit = [&](const uint32_t* k) { return ((KW == 2 && dword == 1 ? k[KW - 1] : k[0]) >> dshift) & 0xFFu; };
#pragma unroll
        for (int i = 0; i < RSC_WARPS * 256 / 4 / RSC_THREADS; ++i)
            reinterpret_cast<uint4*>(s_bins)[i * RSC_THREADS + tid] = make_uint4(0, 0, 0, 0);
        __syncthreads();
#pragma unroll
        for (int i = 0; i < IPT; ++i) {
            if (i < steps) {
                const bool ok = first + i * 32 < count;
                const uint32_t d = digit(key[i]);
                uint32_t peers = __ballot_sync(0xFFFFFFFFu, ok);
#pragma unroll
                for (int b = 0; b < 8; ++b) keep_same_bit(peers, d, 1u << b);
                pos[i] = bins[d] + __popc(peers & below);
                __syncwarp();
                if (ok && (peers >> lane) == 1u) bins[d] = pos[i] + 1u;
                __syncwarp();
            }
        }
        __syncthreads();
        // totals of this CTA to all: a thread takes one bin and half of the warps, then half of the CTAs
        const int b = tid & 255, q = tid >> 8;
        uint32_t sum = 0;
#pragma unroll
        for (int w = 0; w < RSC_WARPS / 2; ++w) sum += s_bins[(q * (RSC_WARPS / 2) + w) * 256 + b];
        s_half[tid] = sum;
        __syncthreads();
        for (int r = q; r < ctas; r += 2) *cluster.map_shared_rank(s_total + rank * 256 + b, r) = s_half[b] + s_half[256 + b];
        cluster.sync();
        if (tid < 256) {
            uint32_t tot = 0, before = 0;
            for (int r = 0; r < ctas; ++r) {
                const uint32_t x = s_total[r * 256 + tid];
                before += r < rank ? x : 0u;
                tot += x;
            }
            uint32_t inc = tot;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t x = __shfl_up_sync(0xFFFFFFFFu, inc, o);
                if (lane >= o) inc += x;
            }
            if (lane == 31) s_warp[warp] = inc;
            s_start[tid] = inc - tot + before;
        }
        __syncthreads();
        uint32_t run = s_start[b] + (q ? s_half[b] : 0u);
        for (int w = 0; w < (b >> 5); ++w) run += s_warp[w];
#pragma unroll
        for (int w = 0; w < RSC_WARPS / 2; ++w) {
            const uint32_t x = s_bins[(q * (RSC_WARPS / 2) + w) * 256 + b];
            s_bins[(q * (RSC_WARPS / 2) + w) * 256 + b] = run;
            run += x;
        }
        __syncthreads();
#pragma unroll
        for (int i = 0; i < IPT; ++i) {
            if (i < steps && first + i * 32 < count) {
                const uint32_t to = bins[digit(key[i])] + pos[i];
                const uint32_t owner = __umulhi(to, cta_rows_inv), at = to - owner * (uint32_t)cta_rows;
                store_key<KW>(cluster.map_shared_rank(s_keys + (size_t)at * KW, owner), key[i]);
                if constexpr (!PACK) *cluster.map_shared_rank(s_vals + at, owner) = val[i];
            }
        }
        cluster.sync();
        if (p == passes - 1) break;
#pragma unroll
        for (int i = 0; i < IPT; ++i) {
            if (i < steps && first + i * 32 < count) {
                load_key<KW>(s_keys + (size_t)(first + i * 32) * KW, key[i]);
                if constexpr (!PACK) val[i] = s_vals[first + i * 32];
            }
        }
    }
    const size_t out = base + row0;
    for (int at = tid; at < count; at += RSC_THREADS) {
        uint32_t id;
        if constexpr (WORDS) {
            id = s_vals[at];
            uint32_t kk[NW];
            load_key<NW>(keys_in + (base + id) * NW, kk);
            store_key<NW>(keys_out + (out + at) * NW, kk);
        } else {
            uint32_t kk[KW];
            load_key<KW>(s_keys + (size_t)at * KW, kk);
            if constexpr (PACK) {
                id = kk[KW - 1] & ((1u << RS_PACK_ID_BITS) - 1u);
                kk[KW - 1] = (kk[0] << (32 - RS_PACK_ID_BITS)) | (kk[KW - 1] >> RS_PACK_ID_BITS);
                kk[0] >>= RS_PACK_ID_BITS;
            } else {
                id = s_vals[at];
            }
            if (compressed) decomp_key<KW>(kk, kc);
            store_key<KW>(keys_out + (out + at) * KW, kk);
        }
        vals_out[out + at] = id;
    }
}

// CTAs that sort a table: 0 when it is not short.  All tables' clusters are to run at once, each CTA on an SM of its own:
// eight CTAs as long as they are three quarters of the SMs (a GPC holds whole clusters only: 16 of eight CTAs
// went in two turns), four up to eight ninths.  A cluster costs 3 us to start and two barriers a pass, which few rows do not
// earn: from 2,048 rows on it pays with packed items (2,000 x 16: 16.9 -> 15.6 us), without from 4,096 with eight
// CTAs (4,000 x 8 in two passes 9.7 -> 9.5, sixteen 63 -> 58) and from 8,192 with four (8,000 x 32: 13.7 -> 14.1 and 99 -> 88,
// 4,000 x 32: 9.7 -> 10.7 and 63 -> 66).  Clusters of two were slower without packed items at every size.
inline int radix_sort_short_ctas(const CtxPtr& c, int n, int L, int NW, bool compressed) {
    // CULSH_SORT_NO_PACK keeps the general form
    const char* no_pack = getenv("CULSH_SORT_NO_PACK");
    if ((no_pack && atoi(no_pack) != 0) || SmallSortCfg<2, true>::SMEM > c->smem_optin) return 0;
    const bool packed = NW == 2 && compressed;
    const int ipt = NW == 2 && !compressed ? SmallSortCfg<2, false>::IPT : SmallSortCfg<1, false>::IPT;
    const int rows = (n + 31) / 32 * 32;  // CTAs hold whole warps of rows
    const int64_t sms = c->sm_count;
    if (L * 8ll * 4 <= sms * 3 && n >= (packed ? 2048 : 4096) && rows <= 8 * RSC_THREADS * ipt) return 8;
    if (L * 4ll * 9 <= sms * 8 && n >= (packed ? 2048 : 8192) && rows <= 4 * RSC_THREADS * ipt) return 4;
    return n <= RSS_THREADS * ipt && L <= sms ? 1 : 0;
}

// keys[0] -> keys[1], row ids to vals[1]
template <int NW, bool PACK>
inline void launch_sort_cluster(const CtxPtr& c, int ctas, uint32_t* keys[2], uint32_t* vals[2], int n, int L, int passes,
                                bool compressed, KeyComp kc, const int* check) {
    constexpr size_t smem = ClusterSortCfg<NW, PACK>::SMEM;
    auto kern = radix_sort_cluster_kernel<NW, PACK>;
    CU_CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    const int cta_rows = (int)ceil_div(ceil_div((size_t)n, (size_t)ctas), 32) * 32;
    const uint32_t inv = 0xFFFFFFFFu / (uint32_t)cta_rows + 1u;  // exact below 2^16 rows of a table
    launch_cluster(c->stream, kern, (unsigned)(L * ctas), (unsigned)ctas, RSC_THREADS, smem, (const uint32_t*)keys[0], keys[1], vals[1], n, cta_rows, inv,
                   passes, compressed, kc, check);
}

template <int NW>
inline int radix_sort_small(const CtxPtr& c, uint32_t* keys[2], uint32_t* vals[2], int n, int L, int passes,
                            bool compressed, KeyComp kc, const int* check) {
    const int ctas = radix_sort_short_ctas(c, n, L, NW, compressed);
    if (ctas > 1) {
        if (c->profiling) cudaEventRecord(c->ev_pass[0], c->stream);
        if (NW == 2 && compressed) launch_sort_cluster<NW, NW == 2>(c, ctas, keys, vals, n, L, passes, compressed, kc, check);
        else launch_sort_cluster<NW, false>(c, ctas, keys, vals, n, L, passes, compressed, kc, check);
        if (c->profiling) cudaEventRecord(c->ev_pass[1], c->stream);
        return 1;
    }
    auto go = [&](auto kern, size_t smem) {
        CU_CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        if (c->profiling) cudaEventRecord(c->ev_pass[0], c->stream);
        launch_next(c->stream, kern, (unsigned)L, RSS_THREADS, smem, keys[0], keys[1], vals[1], n, passes, compressed, kc, check);
        KERNEL_CHECK();
        if (c->profiling) cudaEventRecord(c->ev_pass[1], c->stream);
    };
    if constexpr (NW == 2) {
        if (compressed) go(radix_sort_small_kernel<2, true>, SmallSortCfg<2, true>::SMEM);
        else go(radix_sort_small_kernel<2, false>, SmallSortCfg<2, false>::SMEM);
    } else {
        go(radix_sort_small_kernel<NW, false>, SmallSortCfg<NW, false>::SMEM);
    }
    return 1;
}

// ---------------------------------------------------------------------------------------
// Host driver.  keys[0]/vals[0] hold the input (vals[0] is never read: the first pass
// takes the row id from the position); after radix_sort_passes() passes the result is in
// buffer radix_sort_final(passes, NW).  tile_hist must hold radix_sort_tile_words(n, L, NW) words.
// `compressed` (NW <= 2 only): sort the 5-bit-per-byte form of the keys, see the top of the file.
// ---------------------------------------------------------------------------------------
inline int radix_sort_passes(int KB, bool compressed) { return compressed ? (5 * KB + 7) / 8 : KB; }
inline bool radix_sort_is_small(const CtxPtr& c, int n, int L, int NW, bool compressed) {
    return radix_sort_short_ctas(c, n, L, NW, compressed) > 0;
}
inline int radix_sort_final(const CtxPtr& c, int passes, int n, int L, int NW, bool compressed) {
    return NW >= 4 || radix_sort_is_small(c, n, L, NW, compressed) ? 1 : passes & 1;
}

// Pass step 2 on the host: tile histograms -> destination offsets.  Tables of many tiles leave the bases
// of their chunks behind the tile histograms, [table][chunk][256].
struct TileScan {
    cudaStream_t s;
    int L, tiles_per_table;
    uint32_t* tile_hist;
    bool chunked() const { return tiles_per_table >= RS_CHUNK_MIN_TILES; }
    int n_chunks() const { return chunked() ? (int)ceil_div(tiles_per_table, RS_CHUNK_TILES) : 1; }
    uint32_t* chunk_base() const { return chunked() ? tile_hist + (size_t)tiles_per_table * L * 256 : nullptr; }
    void run() const {
        if (chunked()) {
            launch_next(s, radix_tile_scan_chunk_kernel, (unsigned)(L * n_chunks()), RS_SCAN_THREADS, 0, 
                tile_hist, tiles_per_table, n_chunks(), chunk_base());
            KERNEL_CHECK();
            launch_next(s, radix_chunk_base_kernel, (unsigned)L, 256, 0, chunk_base(), n_chunks());
        } else {
            launch_next(s, radix_tile_scan_kernel, (unsigned)L, RS_SCAN_THREADS, 0, tile_hist, tiles_per_table);
        }
        KERNEL_CHECK();
    }
};

template <int NW>
inline int radix_sort_tables_nw(const CtxPtr& c, uint32_t* keys[2], uint32_t* vals[2], int n, int L,
                                int KB, uint32_t* tile_hist, bool compressed, KeyComp kc) {
    using Cfg = SortCfg<NW>;
    cudaStream_t s = c->stream;
    const int tiles_per_table = (int)ceil_div(n, Cfg::TILE);
    const size_t total_tiles = (size_t)tiles_per_table * L;
    auto k_first = radix_scatter_kernel<NW, true, 0>;
    auto k_next = radix_scatter_kernel<NW, false, 0>;
    auto k_first_c = radix_scatter_kernel<NW, true, 1>;
    auto k_last_c = radix_scatter_kernel<NW, false, 2>;
    constexpr bool CAN_PACK = NW == 2;
    auto k_first_p = radix_scatter_kernel<NW, true, CAN_PACK ? 1 : 0, CAN_PACK>;
    auto k_next_p = radix_scatter_kernel<NW, false, 0, CAN_PACK>;
    auto k_last_p = radix_scatter_kernel<NW, false, CAN_PACK ? 2 : 0, CAN_PACK>;
    // CULSH_SORT_NO_PACK=1 keeps key and id apart in a compressed sort (the tests compare the two)
    const char* no_pack = getenv("CULSH_SORT_NO_PACK");
    const bool pack = compressed && CAN_PACK && n <= (1 << RS_PACK_ID_BITS) && !(no_pack && atoi(no_pack) != 0);
    for (auto k : {k_first, k_next, k_first_c, k_last_c, k_first_p, k_next_p, k_last_p})
        CU_CHECK(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Cfg::SMEM));
    const TileScan scan{s, L, tiles_per_table, tile_hist};
    const int passes = radix_sort_passes(KB, compressed);
    int cur = 0;
    for (int p = 0; p < passes; ++p) {
        if (compressed && p == 0)
            launch_next(s, radix_tile_hist_kernel<NW, true>, (unsigned)total_tiles, RS_THREADS, 0, 
                keys[cur], n, tiles_per_table, p, kc.sub, tile_hist);
        else
            launch_next(s, radix_tile_hist_kernel<NW, false>, (unsigned)total_tiles, RS_THREADS, 0, 
                keys[cur], n, tiles_per_table, pack ? p + 3 : p, 0u, tile_hist);
        KERNEL_CHECK();
        scan.run();
        const bool last = p == passes - 1;
        if (last && c->profiling) cudaEventRecord(c->ev_pass[0], s);
        auto kern = p == 0 ? (compressed ? k_first_c : k_first) : (compressed && last ? k_last_c : k_next);
        if (pack) kern = p == 0 ? k_first_p : (last ? k_last_p : k_next_p);
        launch_next(s, kern, (unsigned)total_tiles, RS_THREADS, Cfg::SMEM, 
            keys[cur], vals[cur], keys[cur ^ 1], vals[cur ^ 1], n, tiles_per_table, p, kc, tile_hist,
            scan.chunk_base(), scan.n_chunks());
        KERNEL_CHECK();
        if (last && c->profiling) cudaEventRecord(c->ev_pass[1], s);
        cur ^= 1;
    }
    return cur;
}

// Keys of NW >= 4 words, word by word from the least significant one: a gather brings the word into the
// order reached so far, up to four passes of the one-word sort order (word, row id) by it, and a last
// gather of whole keys leaves them sorted in keys[1].  keys[0] is only read; the two word arrays live
// in keys[1] until then.  A pass over the keys themselves moves 2 * (4 * NW + 4) bytes per item and
// reads every key again for its histogram: 56 bytes for 16-byte keys, against 20 here and a gather of
// 12 bytes plus a random 32-byte sector per word (the strip of a table, 16 n bytes, is in the L2 for the
// row counts met in practice).
// 2M rows x 32 tables, 16-byte keys: the sort stage 11.2 ms over whole keys, 7.0 this way; 100,003 rows
// x 32: 0.71 -> 0.55.
template <int NW>
inline int radix_sort_words(const CtxPtr& c, uint32_t* keys[2], uint32_t* vals[2], int n, int L, int KB,
                            uint32_t* tile_hist) {
    using Cfg = SortCfg<1>;
    cudaStream_t s = c->stream;
    const int tiles_per_table = (int)ceil_div(n, Cfg::TILE);
    const size_t total_tiles = (size_t)tiles_per_table * L;
    const TileScan scan{s, L, tiles_per_table, tile_hist};
    uint32_t* words[2] = {keys[1], keys[1] + (size_t)n * L};
    auto k_first = radix_scatter_kernel<1, true, 0>;
    auto k_next = radix_scatter_kernel<1, false, 0>;
    auto k_last = radix_scatter_kernel<1, false, 3>;
    for (auto k : {k_first, k_next, k_last})
        CU_CHECK(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Cfg::SMEM));
    // the ids alternate between the two arrays so that the last pass writes vals[1]
    auto ids_of = [&](int pass) { return vals[((KB - 1 - pass) & 1) ? 0 : 1]; };
    for (int p = 0; p < KB; ++p) {
        const bool word_begin = (p & 3) == 0, word_end = (p & 3) == 3 || p == KB - 1;
        const uint32_t* ids = p ? ids_of(p - 1) : nullptr;
        uint32_t* w_in = words[p & 1];
        if (word_begin)
            radix_word_gather_kernel<NW><<<(unsigned)total_tiles, RS_THREADS, 0, s>>>(keys[0], ids, n, tiles_per_table,
                                                                                   NW - 1 - (p >> 2), w_in, tile_hist);
        else
            launch_next(s, radix_tile_hist_kernel<1, false>, (unsigned)total_tiles, RS_THREADS, 0, w_in, n, tiles_per_table, p & 3, 0u, tile_hist);
        KERNEL_CHECK();
        scan.run();
        if (p == KB - 1 && c->profiling) cudaEventRecord(c->ev_pass[0], s);
        auto kern = p == 0 ? k_first : (word_end ? k_last : k_next);  // a key has nine bytes at least
        launch_next(s, kern, (unsigned)total_tiles, RS_THREADS, Cfg::SMEM, w_in, ids, words[(p & 1) ^ 1], ids_of(p), n, tiles_per_table, p & 3,
                                                               KeyComp{0u, 0u}, tile_hist, scan.chunk_base(), scan.n_chunks());
        KERNEL_CHECK();
        if (p == KB - 1 && c->profiling) cudaEventRecord(c->ev_pass[1], s);
    }
    const int gather_tiles = (int)ceil_div((size_t)n * (NW / 4), RS_THREADS * 8);
    radix_key_gather_kernel<NW><<<(unsigned)((size_t)gather_tiles * L), RS_THREADS, 0, s>>>(keys[0], vals[1], n, gather_tiles, keys[1]);
    KERNEL_CHECK();
    return 1;
}

inline size_t radix_sort_tile_words(int n, int L, int NW) {
    const size_t tiles = ceil_div(n, sort_tile_items(NW));
    return (tiles + ceil_div(tiles, (size_t)RS_CHUNK_TILES)) * (size_t)L * 256;  // tile histograms + chunk totals
}

inline int radix_sort_tables(const CtxPtr& c, int NW, uint32_t* keys[2], uint32_t* vals[2], int n,
                             int L, int KB, uint32_t* tile_hist, bool compressed = false,
                             KeyComp kc = KeyComp{0u, 0u}, const int* check = nullptr) {
    if (radix_sort_is_small(c, n, L, NW, compressed)) {
        const int passes = radix_sort_passes(KB, compressed);
        switch (NW) {
            case 1: return radix_sort_small<1>(c, keys, vals, n, L, passes, compressed, kc, check);
            case 2: return radix_sort_small<2>(c, keys, vals, n, L, passes, compressed, kc, check);
            case 4: return radix_sort_small<4>(c, keys, vals, n, L, passes, compressed, kc, check);
            case 8: return radix_sort_small<8>(c, keys, vals, n, L, passes, compressed, kc, check);
            case 16: return radix_sort_small<16>(c, keys, vals, n, L, passes, compressed, kc, check);
        }
    }
    switch (NW) {
        case 1: return radix_sort_tables_nw<1>(c, keys, vals, n, L, KB, tile_hist, compressed, kc);
        case 2: return radix_sort_tables_nw<2>(c, keys, vals, n, L, KB, tile_hist, compressed, kc);
        case 4: return radix_sort_words<4>(c, keys, vals, n, L, KB, tile_hist);
        case 8: return radix_sort_words<8>(c, keys, vals, n, L, KB, tile_hist);
        case 16: return radix_sort_words<16>(c, keys, vals, n, L, KB, tile_hist);
    }
    fail(CULSH_ERR_UNSUPPORTED, "unsupported key width: %d words", NW);
}

// ---------------------------------------------------------------------------------------
// Device-wide exclusive scan.  out has n+1 elements: out[n] = total.  The sums of its blocks, then the blocks; up to
// SCAN_ADD_MAX blocks a block adds up the sums before its own itself, more of them are scanned in a launch between
// the two (100,003 elements: 12 us in three launches, 8.6 in two).  What a block adds grows with its number: the line lies where that
// is four reads a thread.  Three launches and two, 64-bit elements: 64 blocks 13.4 and 10.3 us, 1,024 23.8 and 20.7, 8,192 138 and 135.
// ---------------------------------------------------------------------------------------
constexpr int SCAN_THREADS = 256;
constexpr int SCAN_IPT = 8;
constexpr int SCAN_TILE = SCAN_THREADS * SCAN_IPT;
constexpr size_t SCAN_ADD_MAX = 1024;

template <typename TOut>
__device__ __forceinline__ TOut block_exclusive_scan(TOut v, TOut* s_warp, TOut& total) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    TOut inc = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        TOut x = __shfl_up_sync(0xFFFFFFFFu, inc, o);
        if (lane >= o) inc += x;
    }
    __syncthreads();  // protect s_warp reuse between calls
    if (lane == 31) s_warp[w] = inc;
    __syncthreads();
    TOut base = 0, tot = 0;
    const int nw = blockDim.x >> 5;
    for (int i = 0; i < nw; ++i) {
        TOut x = s_warp[i];
        if (i < w) base += x;
        tot += x;
    }
    total = tot;
    return base + inc - v;
}

template <typename TIn, typename TOut>
__global__ void __launch_bounds__(SCAN_THREADS)
scan_reduce_kernel(const TIn* __restrict__ in, size_t n, TOut* __restrict__ block_sums, KernelBefore kernel_before) {
    behind_kernel_before(in, block_sums, kernel_before);
    __shared__ TOut s_warp[32];
    size_t base = (size_t)blockIdx.x * SCAN_TILE;
    TOut sum = 0;
    for (int i = 0; i < SCAN_IPT; ++i) {
        size_t idx = base + (size_t)i * SCAN_THREADS + threadIdx.x;
        if (idx < n) sum += (TOut)in[idx];
    }
    TOut total;
    block_exclusive_scan<TOut>(sum, s_warp, total);
    if (threadIdx.x == 0) block_sums[blockIdx.x] = total;
}

// What a scan leaves in page-locked host memory besides its result: its total and a few 32-bit words from elsewhere.  The
// host reads them behind its next wait; as a copy of its own each of them cost 3 us on the device and as much
// in between.
struct HostWords {
    uint64_t* total;       // or null: nothing
    uint32_t* words;       // [n_a + n_b]
    const uint32_t *a, *b;
    int n_a, n_b;
    __device__ __forceinline__ void write(uint64_t t) const { write(t, a); }
    // By one warp.  `from` in place of a: a kernel that makes these words itself writes the array that a is, through another pointer.
    __device__ __forceinline__ void write(uint64_t t, const uint32_t* from) const {
        if (!total) return;
        const int i = threadIdx.x & 31;
        if (i == 0) *total = t;
        if (i < n_a) words[i] = from[i];
        else if (i < n_a + n_b) words[i] = b[i - n_a];
    }
};

template <typename TOut>
__global__ void __launch_bounds__(1024)
scan_block_sums_kernel(TOut* __restrict__ block_sums, size_t n_blocks, TOut* __restrict__ total_out, HostWords host, KernelBefore kernel_before) {
    behind_kernel_before(block_sums, total_out, kernel_before);
    __shared__ TOut s_warp[32];
    TOut carry = 0;
    for (size_t base = 0; base < n_blocks; base += 1024) {
        size_t idx = base + threadIdx.x;
        TOut v = idx < n_blocks ? block_sums[idx] : TOut(0);
        TOut total;
        TOut ex = block_exclusive_scan<TOut>(v, s_warp, total);
        if (idx < n_blocks) block_sums[idx] = carry + ex;
        carry += total;
    }
    if (threadIdx.x == 0 && total_out) *total_out = carry;
    if (threadIdx.x < 32) host.write((uint64_t)carry);
}

template <typename TIn, typename TOut>
__global__ void __launch_bounds__(SCAN_THREADS)
scan_apply_kernel(const TIn* __restrict__ in, size_t n, const TOut* __restrict__ block_sums, bool scanned,
                  TOut* __restrict__ out, HostWords host, KernelBefore kernel_before) {
    behind_kernel_before(in, block_sums, out, kernel_before);
    __shared__ TOut s_warp[32];
    TOut before = 0;  // elements of the blocks before this one
    if (scanned) {
        before = block_sums[blockIdx.x];
    } else {
        TOut sum = 0;
        for (unsigned i = threadIdx.x; i < blockIdx.x; i += SCAN_THREADS) sum += block_sums[i];
        block_exclusive_scan<TOut>(sum, s_warp, before);
    }
    const size_t base = (size_t)blockIdx.x * SCAN_TILE + (size_t)threadIdx.x * SCAN_IPT;
    TOut v[SCAN_IPT];
    TOut sum = 0;
#pragma unroll
    for (int i = 0; i < SCAN_IPT; ++i) {
        size_t idx = base + i;
        v[i] = idx < n ? (TOut)in[idx] : TOut(0);
        sum += v[i];
    }
    TOut total;
    TOut ex = block_exclusive_scan<TOut>(sum, s_warp, total) + before;
    if (!scanned && blockIdx.x == gridDim.x - 1) {
        if (threadIdx.x == 0) out[n] = before + total;
        if (threadIdx.x < 32) host.write((uint64_t)(before + total));
    }
#pragma unroll
    for (int i = 0; i < SCAN_IPT; ++i) {
        size_t idx = base + i;
        if (idx < n) out[idx] = ex;
        ex += v[i];
    }
}

// Short arrays: one CTA walks the array in steps of 4096 elements and carries the total along.  A step takes about 3 us
// as long as a warp's accesses are 16 bytes a lane (with eight words a lane, one access each, it was 4: every access met
// 16 lines), two launches 8 whatever the size.
constexpr int SCAN_ONE_THREADS = 1024;
constexpr int SCAN_ONE_IPT = 4;
constexpr int SCAN_ONE_STEP = SCAN_ONE_THREADS * SCAN_ONE_IPT;
constexpr size_t SCAN_ONE_MAX = 2 * SCAN_ONE_STEP;

template <typename T>
struct alignas(16) ScanVec {
    T v[16 / sizeof(T)];
};

// in and out on 16-byte boundaries
template <typename T>
__global__ void __launch_bounds__(SCAN_ONE_THREADS)
scan_one_kernel(const T* __restrict__ in, int n, T* __restrict__ out, HostWords host, KernelBefore kernel_before) {
    behind_kernel_before(in, out, kernel_before);
    constexpr int PER = 16 / sizeof(T), VECS = SCAN_ONE_IPT / PER;
    __shared__ T s_warp[32];
    T carry = 0;
    for (int base = 0; base < n; base += SCAN_ONE_STEP) {
        const int first = base + threadIdx.x * SCAN_ONE_IPT;
        const bool whole = first + SCAN_ONE_IPT <= n;
        ScanVec<T> v[VECS];
        T sum = 0;
#pragma unroll
        for (int i = 0; i < VECS; ++i) {
            if (whole) v[i] = reinterpret_cast<const ScanVec<T>*>(in + first)[i];
#pragma unroll
            for (int j = 0; j < PER; ++j) {
                const int at = first + i * PER + j;
                if (!whole) v[i].v[j] = at < n ? in[at] : T(0);
                sum += v[i].v[j];
            }
        }
        T total;
        T ex = block_exclusive_scan<T>(sum, s_warp, total) + carry;
#pragma unroll
        for (int i = 0; i < VECS; ++i) {
#pragma unroll
            for (int j = 0; j < PER; ++j) {
                const T x = v[i].v[j];
                v[i].v[j] = ex;
                ex += x;
                const int at = first + i * PER + j;
                if (!whole && at < n) out[at] = v[i].v[j];
            }
            if (whole) reinterpret_cast<ScanVec<T>*>(out + first)[i] = v[i];
        }
        carry += total;
    }
    if (threadIdx.x == 0) out[n] = carry;
    if (threadIdx.x < 32) host.write((uint64_t)carry);
}

// scratch must hold ceil(n / SCAN_TILE) TOut elements.  out[n] receives the total.  `host` needs n > 0.
template <typename TIn, typename TOut>
inline void exclusive_scan(cudaStream_t s, const TIn* in, size_t n, TOut* out, TOut* scratch, const HostWords& host = HostWords{}) {
    if (n == 0) {
        CU_CHECK(cudaMemsetAsync(out, 0, sizeof(TOut), s));
        return;
    }
    if constexpr (std::is_same<TIn, TOut>::value) {
        if (n <= SCAN_ONE_MAX && ((reinterpret_cast<uintptr_t>(in) | reinterpret_cast<uintptr_t>(out)) & 15) == 0) {
            launch_next(s, scan_one_kernel<TOut>, 1, SCAN_ONE_THREADS, 0, in, (int)n, out, host);
            KERNEL_CHECK();
            return;
        }
    }
    size_t n_blocks = ceil_div(n, SCAN_TILE);
    launch_next(s, scan_reduce_kernel<TIn, TOut>, (unsigned)n_blocks, SCAN_THREADS, 0, in, n, scratch);
    KERNEL_CHECK();
    const bool scanned = n_blocks > SCAN_ADD_MAX;
    if (scanned) {
        launch_next(s, scan_block_sums_kernel<TOut>, 1, 1024, 0, scratch, n_blocks, out + n, host);
        KERNEL_CHECK();
    }
    launch_next(s, scan_apply_kernel<TIn, TOut>, (unsigned)n_blocks, SCAN_THREADS, 0, in, n, scratch, scanned, out, host);
    KERNEL_CHECK();
}

inline size_t scan_scratch_elems(size_t n) { return ceil_div(n, SCAN_TILE) + 1; }

}  // namespace culsh_b200
