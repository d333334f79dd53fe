// Query side: bucket lookup, candidate gather and per-query cross-table dedupe, written
// into the CSR result.  Replaces find_matching_buckets_kernel (core/query.cuh:31-101) and
// query_from_matched_buckets (core/query.cuh:290-478): upstream materialises the raw
// candidates, runs a 32-bit segmented radix sort over them, flags/reduces/scans and
// compacts (about 15 passes over `raw` ints); here each query's bucket lists are merged
// on chip - a shared-memory bitmap over row ids for large candidate sets, a warp-level
// sort for small ones - and each list is read once, its unique ids written to the query's raw span and copied from there.
#pragma once

#include "common.cuh"
#include "index_build.cuh"
#include "radix_sort.cuh"

namespace culsh_b200 {

// ---------------------------------------------------------------------------------------
// Lookup: one thread per (table, query); binary search over the table's sorted bucket keys.
// ---------------------------------------------------------------------------------------
template <int NW>
__device__ __forceinline__ int compare_keys(const uint32_t* __restrict__ a,
                                            const uint32_t* __restrict__ b) {
#pragma unroll
    for (int w = 0; w < NW; ++w) {
        if (a[w] != b[w]) return a[w] < b[w] ? -1 : 1;
    }
    return 0;
}

// bounds[t*n_q + q] = the matched bucket's list [x, y) in `cand`, (0, 0) when there is none.  Table
// major, like the query keys: neighbouring threads (queries) read and write neighbouring words here,
// in the count and in the warp path, and a self-join writes the same array from its buckets.
//
// One thread for a pair, or `group` neighbouring lanes (a power of two), each looking at a bucket of its own in every step, so that a step leaves
// 1 / (group + 1) of them: idx is that of the group's pair then, `have` whether it has one, and whole warps call.
template <int NW>
__device__ __forceinline__ int2 lookup_pair(const uint32_t* __restrict__ qkeys, const uint8_t* __restrict__ q_ovf, int n_q,
                                            size_t idx, const uint32_t* __restrict__ bucket_keys,
                                            const int32_t* __restrict__ bucket_offsets, const int32_t* __restrict__ table_offsets) {
    const int t = (int)(idx / n_q);
    uint32_t key[NW];
    load_key<NW>(qkeys + idx * NW, key);
    int lo = table_offsets[t], hi = table_offsets[t + 1] - 1;
    int2 found = make_int2(0, 0);
    if (q_ovf && q_ovf[idx]) hi = lo - 1;  // value outside the index's narrow range: no bucket
    while (lo <= hi) {
        int mid = lo + ((hi - lo) >> 1);
        int c = compare_keys<NW>(key, bucket_keys + (size_t)mid * NW);
        if (c == 0) { found = make_int2(bucket_offsets[mid], bucket_offsets[mid + 1]); break; }
        if (c < 0) hi = mid - 1; else lo = mid + 1;
    }
    return found;
}
template <int NW>
__device__ __forceinline__ int2 lookup_pair_together(const uint32_t* __restrict__ qkeys, const uint8_t* __restrict__ q_ovf, int n_q,
                                            size_t idx, bool have, int group, const uint32_t* __restrict__ bucket_keys,
                                            const int32_t* __restrict__ bucket_offsets, const int32_t* __restrict__ table_offsets) {
    const int lane = threadIdx.x & 31, at = lane & (group - 1), first = lane - at;
    const uint32_t mine = (group == 32 ? 0xFFFFFFFFu : (1u << group) - 1u) << first;
    uint32_t key[NW];
    int lo = 0, hi = 0, found = -1;
    if (have) {
        const int t = (int)(idx / n_q);
        load_key<NW>(qkeys + idx * NW, key);
        lo = table_offsets[t];
        hi = table_offsets[t + 1];
        if (q_ovf && q_ovf[idx]) hi = lo;  // value outside the index's narrow range: no bucket
    }
    while (__any_sync(0xFFFFFFFFu, lo < hi)) {
        const int len = hi - lo;
        const bool few = len <= group;
        auto place = [&](int i) { return few ? lo + i : lo + (int)((int64_t)(i + 1) * len / (group + 1)); };
        int c = 1;  // of the bucket and the key
        if (few ? at < len : lo < hi) c = compare_keys<NW>(bucket_keys + (size_t)place(at) * NW, key);
        const uint32_t below = __ballot_sync(0xFFFFFFFFu, c < 0) & mine, same = __ballot_sync(0xFFFFFFFFu, c == 0) & mine;
        if (lo < hi) {
            const int n = __popc(below);  // the first n of them
            if (same) {
                found = place(__ffs(same) - 1 - first);
                hi = lo;
            } else if (few) {
                hi = lo;
            } else {
                const int end = n < group ? place(n) : hi;
                if (n > 0) lo = place(n - 1) + 1;
                hi = end;
            }
        }
    }
    return found < 0 ? make_int2(0, 0) : make_int2(bucket_offsets[found], bucket_offsets[found + 1]);
}

// A CTA takes a stretch of the queries of one table.  A search is a chain of dependent
// reads that neighbouring threads do not share, about eighteen in a table of 260,000 buckets: keys of the table, evenly
// spread, as many as the CTA's threads read words, come into shared memory first and take the upper levels out of the
// chain, eight of them with keys of one word (10,000 queries x 32 tables of 1M rows 15.6 -> 12.5 us, 100,003 x 24: 89 -> 85,
// 10,000 x 32 with keys of four words 78 -> 70; 1,024 keys and four queries a thread: 102 in place of 85).
constexpr int LU_THREADS = 256;
template <int NW>
__global__ void __launch_bounds__(LU_THREADS)
lookup_kernel(const uint32_t* __restrict__ qkeys, const uint8_t* __restrict__ q_ovf, int n_q, int chunks,
              const uint32_t* __restrict__ bucket_keys, const int32_t* __restrict__ bucket_offsets,
              const int32_t* __restrict__ table_offsets, int2* __restrict__ bounds, KernelBefore kernel_before) {
    behind_kernel_before(qkeys, q_ovf, bucket_keys, bucket_offsets, table_offsets, bounds, kernel_before);
    constexpr int SPLIT = LU_THREADS / NW;  // a power of two
    __shared__ __align__(16) uint32_t s_split[SPLIT * NW];
    const int t = blockIdx.x / chunks;
    const int64_t q = (int64_t)(blockIdx.x - t * chunks) * LU_THREADS + threadIdx.x;
    const size_t idx = (size_t)t * n_q + q;
    const int first = table_offsets[t], n_b = table_offsets[t + 1] - first;
    const int step = n_b / SPLIT + 1;                // buckets from one split to the next
    const int n_split = (n_b + step - 1) / step;     // split i is bucket first + i * step
    const uint32_t* keys = bucket_keys + (size_t)first * NW;
    uint32_t key[NW];
    if (q < n_q) load_key<NW>(qkeys + idx * NW, key);
    if (threadIdx.x < n_split) {
        uint32_t k[NW];
        load_key<NW>(keys + (size_t)threadIdx.x * step * NW, k);
        store_key<NW>(s_split + threadIdx.x * NW, k);
    }
    __syncthreads();
    if (q >= n_q) return;
    int2 found = make_int2(0, 0);
    int at = 0;  // splits at or below the key
#pragma unroll
    for (int s = SPLIT; s > 0; s >>= 1)
        if (at + s <= n_split && compare_keys<NW>(s_split + (at + s - 1) * NW, key) <= 0) at += s;
    if (at > 0 && !(q_ovf && q_ovf[idx])) {  // a value outside the index's narrow range has no bucket
        bool same = compare_keys<NW>(s_split + (at - 1) * NW, key) == 0;
        // the last bucket at or below the key, from the one of the split on
        int lo = (at - 1) * step, hi = min(n_b - lo, step) + lo - 1;
        while (!same && lo < hi) {
            const int mid = hi - ((hi - lo) >> 1);  // above lo
            const int c = compare_keys<NW>(keys + (size_t)mid * NW, key);
            if (c <= 0) {
                lo = mid;
                same = c == 0;
            } else {
                hi = mid - 1;
            }
        }
        if (same) found = make_int2(bucket_offsets[first + lo], bucket_offsets[first + lo + 1]);
    }
    bounds[idx] = found;
}

template <int NW>
inline void launch_lookup(const CtxPtr& c, const uint32_t* qkeys, const uint8_t* q_ovf, int n_q, int L, const uint32_t* bucket_keys,
                          const int32_t* bucket_offsets, const int32_t* table_offsets, int2* bounds) {
    const int chunks = (int)ceil_div(n_q, LU_THREADS);
    launch_next(c->stream, lookup_kernel<NW>, (unsigned)((size_t)chunks * L), LU_THREADS, 0, qkeys, q_ovf, n_q, chunks, bucket_keys,
                                                                                  bucket_offsets, table_offsets, bounds);
    KERNEL_CHECK();
}

// ---------------------------------------------------------------------------------------
// Raw (pre-dedupe) candidate count per query; queries above the small-path limit are
// appended to big_list.  In a self-join every list of two or more rows holds the query's own row
// and lists of that row alone are not in `bounds` at all, so the row is counted once and taken
// off every list: the count is what the result can hold at most.
// ---------------------------------------------------------------------------------------
// largest raw count handled by the warp path (1024: 32 ids per lane in the sort network; with 512
// the queries of 513 - 1024 ids of a 12.5M-row shard took a CTA each on the sort path: 0.77 -> 0.50 ms
// per 10k queries, the 10M-row self-join, all below 512, is unchanged)
constexpr int SMALL_MAX = 1024;
// ... and by its short form (4 ids per lane: 512 bytes of shared memory a warp and 40 registers, so that 48 of an
// SM's 64 warp slots are filled; the long form, 64 registers, fills 32)
constexpr int SHORT_MAX = 128;

// rows of a packed list other than the query's own
__device__ __forceinline__ uint32_t packed_count(const BoundsView& bounds, int t, uint32_t w) {
    if (w == 0) return 0;
    if (w & PB_PAIR) return 1;
    const int2 b = bounds.unpack(t, w);
    return (uint32_t)(b.y - b.x) - 1u;
}

constexpr int RC_BATCH = 8;
// counters[0] = queries for the bitmap path (big_list), counters[1] = queries for the
// shared-memory sort path (mid_list; only used when mid_max > SMALL_MAX), counters[2] = queries for
// the long form of the warp path
__global__ void __launch_bounds__(256)
raw_count_kernel(BoundsView bounds, int n_q, int L, bool self_join, uint64_t* __restrict__ raw_cnt,
                 uint32_t* __restrict__ big_list, uint32_t* __restrict__ mid_list, uint32_t* __restrict__ counters,
                 int mid_max, uint64_t* __restrict__ uniq_cnt, KernelBefore kernel_before) {
    behind_kernel_before(raw_cnt, big_list, mid_list, counters, uniq_cnt, kernel_before);
    const uint32_t q = blockIdx.x * blockDim.x + threadIdx.x;  // unsigned: the last CTA may reach past 2^31
    if (q >= (uint32_t)n_q) return;
    uint32_t c = self_join ? 1u : 0u;  // at most n * L < 2^31
    int t = 0;
    for (; t + RC_BATCH <= L; t += RC_BATCH) {  // RC_BATCH loads in flight
        if (bounds.pair) {
            int2 b[RC_BATCH];
#pragma unroll
            for (int j = 0; j < RC_BATCH; ++j) b[j] = bounds.pair[(size_t)(t + j) * n_q + q];
#pragma unroll
            for (int j = 0; j < RC_BATCH; ++j) c += (uint32_t)(b[j].y - b[j].x);
        } else {
            uint32_t w[RC_BATCH];
#pragma unroll
            for (int j = 0; j < RC_BATCH; ++j) w[j] = bounds.packed[(size_t)(t + j) * n_q + q];
#pragma unroll
            for (int j = 0; j < RC_BATCH; ++j) {
                c += packed_count(bounds, t + j, w[j]);
            }
        }
    }
    for (; t < L; ++t) {
        if (bounds.pair) {
            const int2 b = bounds.pair[(size_t)t * n_q + q];
            c += (uint32_t)(b.y - b.x);
        } else {
            c += packed_count(bounds, t, bounds.packed[(size_t)t * n_q + q]);
        }
    }
    raw_cnt[q] = c;
    if (c > SMALL_MAX) {
        uniq_cnt[q] = 0;  // its windows add up in it
        // the sort path gathers a self-join's lists with the own row in each
        if (c + (self_join ? (uint32_t)L : 0u) <= (uint32_t)mid_max) mid_list[atomicAdd(&counters[1], 1u)] = q;
        else big_list[atomicAdd(&counters[0], 1u)] = q;
    } else if (c > SHORT_MAX) {
        atomicAdd(&counters[2], 1u);
    }
}

// Few (table, query) pairs: lookup, raw counts, their scan and the counters in one launch
// in place of five (memset, lookup, count, scan; one query against 32 tables, the whole call: 153 -> 143 us).  A thread's search is
// a chain of about twenty dependent reads of lines of their own: as many lanes as there are threads for it share one, up to a warp (1M rows, the whole
// call with a thread and with a warp: 32 pairs 75 and 66 us, 1,024 74 and 67; eight lanes as good as 32, four 1 us worse; two lanes 2 to 4 us slower than one).  Above
// LS_ONE_PAIRS a cluster of eight CTAs shares the pairs and adds the counts up in the shared memory of its first CTA, which does the rest; it
// starts 2 us later than one CTA, whose SM can have so many reads in flight (512 pairs in one CTA 75 us, 1,024 in the cluster 67).  Up to 8,192 pairs
// the call as a whole is faster this way than with a launch for each step (1M rows x 32 tables, 2,080 pairs 71.3 -> 64.0 us, 8,192 86 ->
// 67; 10M rows 102 -> 80 and 89 -> 85).
constexpr int LS_THREADS = 1024;
constexpr int LS_CTAS = 8;
constexpr size_t LS_ONE_PAIRS = 128;
constexpr size_t LS_MAX_PAIRS = LS_CTAS * LS_THREADS;
constexpr int LS_GROUP = 32;  // lanes that search for a pair, at most
template <int NW>
__global__ void __launch_bounds__(LS_THREADS)
lookup_count_kernel(const uint32_t* __restrict__ qkeys, const uint8_t* __restrict__ q_ovf, int n_q, int L,
                    const uint32_t* __restrict__ bucket_keys, const int32_t* __restrict__ bucket_offsets,
                    const int32_t* __restrict__ table_offsets, int2* __restrict__ bounds, uint64_t* __restrict__ raw_cnt,
                    uint64_t* __restrict__ raw_off, uint32_t* __restrict__ big_list, uint32_t* __restrict__ mid_list,
                    uint32_t* __restrict__ counters, int mid_max, uint64_t* __restrict__ uniq_cnt, int group, HostWords host, KernelBefore kernel_before) {
    behind_kernel_before(qkeys, q_ovf, bucket_keys, bucket_offsets, table_offsets, bounds, raw_cnt, raw_off, big_list, mid_list, counters, uniq_cnt, kernel_before);
    __shared__ uint32_t s_cnt[LS_MAX_PAIRS];  // at most as many queries as pairs
    __shared__ uint32_t s_counters[3];
    __shared__ uint64_t s_warp[32];
    const int tid = threadIdx.x;
    for (int q = tid; q < n_q; q += LS_THREADS) s_cnt[q] = 0;
    if (tid < 3) s_counters[tid] = 0;
    __syncthreads();
    auto cluster = cooperative_groups::this_cluster();
    const int rank = (int)cluster.block_rank(), share = (n_q * L + (int)cluster.num_blocks() - 1) / (int)cluster.num_blocks();
    uint32_t* const cnt = cluster.map_shared_rank(s_cnt, 0);
    cluster.sync();
    const int end = min(n_q * L, (rank + 1) * share), at_once = LS_THREADS / group;
    for (int first = rank * share; first < end; first += at_once) {
        const int idx = first + tid / group;
        const bool have = idx < end;
        int2 b = make_int2(0, 0);
        if (group > 1) b = lookup_pair_together<NW>(qkeys, q_ovf, n_q, idx, have, group, bucket_keys, bucket_offsets, table_offsets);
        else if (have) b = lookup_pair<NW>(qkeys, q_ovf, n_q, idx, bucket_keys, bucket_offsets, table_offsets);
        if (have && tid % group == 0) {
            bounds[idx] = b;
            if (b.y > b.x) atomicAdd(cnt + idx % n_q, (uint32_t)(b.y - b.x));
        }
    }
    cluster.sync();
    if (rank > 0) return;
    uint64_t carry = 0;
    for (int q0 = 0; q0 < n_q; q0 += LS_THREADS) {
        const int q = q0 + tid;
        const uint32_t c = q < n_q ? s_cnt[q] : 0u;
        uint64_t total;
        const uint64_t ex = block_exclusive_scan<uint64_t>((uint64_t)c, s_warp, total);
        if (q < n_q) {
            raw_cnt[q] = c;
            raw_off[q] = carry + ex;
            if (c > SMALL_MAX) {
                uniq_cnt[q] = 0;
                if (c <= (uint32_t)mid_max) mid_list[atomicAdd(&s_counters[1], 1u)] = (uint32_t)q;
                else big_list[atomicAdd(&s_counters[0], 1u)] = (uint32_t)q;
            } else if (c > SHORT_MAX) {
                atomicAdd(&s_counters[2], 1u);
            }
        }
        carry += total;
    }
    __syncthreads();
    if (tid == 0) raw_off[n_q] = carry;
    if (tid < 3) counters[tid] = s_counters[tid];
    if (tid < 32) host.write(carry, s_counters);
}

// ---------------------------------------------------------------------------------------
// Small path: one warp per query, raw <= SMALL_MAX.  The ids are gathered into the warp's slice
// of shared memory, sorted in registers (bitonic, shuffles), made unique and compacted by
// ballots.  Output goes to tmp[raw_off[q] ...].
// ---------------------------------------------------------------------------------------
constexpr int SM_THREADS = 256;
constexpr int SM_WARPS = SM_THREADS / 32;

// Bitonic sort of 32*E ids, position p = E*lane + e in v[e] of `lane`, then adjacent-unique and
// ballot compaction to out[]; returns the number of unique ids.  Exchanges at distance < E stay
// inside a lane, the others are one shuffle and one min / max each.  Every merge starts with the
// reversing step (partner p ^ (size - 1)), after which all steps go upwards, so that which of the
// two a lane keeps is one bit of its number.  The network is what the warp path spends its
// instructions on: with the striped layout (p = 32*e + lane) and alternating directions it took 190
// instructions for 64 ids instead of 80 and the gather of the 10M-row self-join 8.9 ms instead of 6.3.
template <int E>
__device__ __forceinline__ int warp_sort_unique(const int32_t* __restrict__ buf, int r, int lane,
                                                int32_t* __restrict__ out) {
    int32_t v[E];
#pragma unroll
    for (int e = 0; e < E; ++e) {  // which id starts where does not matter: the striped read has no bank conflicts
        const int p = 32 * e + lane;
        v[e] = p < r ? buf[p] : 0x7FFFFFFF;
    }
#pragma unroll
    for (int ksz = 2; ksz <= 32 * E; ksz <<= 1) {
        if (ksz <= E) {  // reversing step inside the lane
#pragma unroll
            for (int e = 0; e < E; ++e) {
                const int f = e ^ (ksz - 1);
                if (e < f) {
                    const int32_t a = v[e], b = v[f];
                    v[e] = min(a, b);
                    v[f] = max(a, b);
                }
            }
        } else {  // partner lane ^ (ksz / E - 1), its ids in reverse order
            const bool low = (lane & (ksz / (2 * E))) == 0;
            int32_t o[E];
#pragma unroll
            for (int e = 0; e < E; ++e) o[e] = __shfl_xor_sync(0xFFFFFFFFu, v[E - 1 - e], ksz / E - 1);
#pragma unroll
            for (int e = 0; e < E; ++e) v[e] = low ? min(v[e], o[e]) : max(v[e], o[e]);
        }
#pragma unroll
        for (int j = ksz >> 2; j > 0; j >>= 1) {
            if (j >= E) {
                const bool low = (lane & (j / E)) == 0;
#pragma unroll
                for (int e = 0; e < E; ++e) {
                    const int32_t other = __shfl_xor_sync(0xFFFFFFFFu, v[e], j / E);
                    v[e] = low ? min(v[e], other) : max(v[e], other);
                }
            } else {
#pragma unroll
                for (int e = 0; e < E; ++e) {
                    if ((e & j) == 0) {
                        const int32_t a = v[e], b = v[e | j];
                        v[e] = min(a, b);
                        v[e | j] = max(a, b);
                    }
                }
            }
        }
    }
    // ids below the first padding value that differ from their predecessor
    int32_t prev = __shfl_up_sync(0xFFFFFFFFu, v[E - 1], 1);
    if (lane == 0) prev = -1;
    int mine = 0;
    uint32_t keep = 0;
#pragma unroll
    for (int e = 0; e < E; ++e) {
        if (v[e] != prev && v[e] != 0x7FFFFFFF) { keep |= 1u << e; ++mine; }
        prev = v[e];
    }
    int inc = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int x = __shfl_up_sync(0xFFFFFFFFu, inc, o);
        if (lane >= o) inc += x;
    }
    int32_t* dst = out + (inc - mine);
#pragma unroll
    for (int e = 0; e < E; ++e)
        if (keep & (1u << e)) *dst++ = v[e];
    return __shfl_sync(0xFFFFFFFFu, inc, 31);
}

// An id into the warp's buffer at dst.  SELF: without the query's own row, which a list holds once (the
// ids behind it move up by one).
template <bool SELF>
__device__ __forceinline__ void put_id(int32_t* __restrict__ buf, int dst, int32_t x, int q) {
    if (!SELF) buf[dst] = x;
    else if (x != q) buf[dst - (x > q ? 1 : 0)] = x;
}

// The ids of 64 lists: each lane fetches the first four of two lists with independent loads, and what longer lists
// hold beyond these is laid end to end and fetched by the whole warp, SM_LOADS ids a lane in flight.  List after
// list, with the loads of one list in flight, a query waited for memory once for each long list (100,003 queries of 24
// lists and 170 ids: 200 us, 173 this way).  A self-join keeps that order: its longer lists are few (10M rows x 48 tables, all
// lists in one: 7.3 -> 9.3 ms; 100,003 rows with sets of up to 1,024: 242 -> 280 us).
constexpr int SM_LOADS = 8;
struct WarpLists {
    int32_t pre[65];   // ids beyond the fourth, of the lists before this one; [64] all of them
    int32_t src[64];   // id p of that sequence is cand[src + p]
    int32_t dst[64];   // and goes to buf[dst + p]
};

// Takes the queries with `above` < raw <= CAP (and with `above` = 0 the empty ones).  Nothing is done when all of them
// together have more than `room` ids: a launch whose counts the host has not seen says how many `tmp` holds.
template <int CAP, bool SELF>
__global__ void __launch_bounds__(SM_THREADS, CAP == SHORT_MAX ? 6 : 4)
dedupe_small_kernel(BoundsView bounds, const int32_t* __restrict__ cand, const uint64_t* __restrict__ raw_cnt,
                    const uint64_t* __restrict__ raw_off, int L, int above, uint64_t room, int32_t* __restrict__ tmp,
                    uint64_t* __restrict__ uniq_cnt, KernelBefore kernel_before) {
    behind_kernel_before(cand, raw_cnt, raw_off, tmp, uniq_cnt, kernel_before);
    __shared__ int32_t s_buf[SM_WARPS][CAP];
    __shared__ WarpLists s_lists[SELF ? 1 : SM_WARPS];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int n_q = bounds.n_q;
    int32_t* buf = s_buf[warp];
    WarpLists& wl = s_lists[SELF ? 0 : warp];
    if (raw_off[n_q] > room) return;
    for (uint32_t qu = blockIdx.x * SM_WARPS + warp; qu < (uint32_t)n_q; qu += gridDim.x * SM_WARPS) {
        const int q = (int)qu;
        const uint64_t r64 = raw_cnt[q];
        if (r64 > CAP) continue;  // another launch owns it
        const int r = (int)r64;
        if (above && r <= above) continue;
        if (r == 0) {
            if (lane == 0) uniq_cnt[q] = 0;
            continue;
        }
        // Gather the bucket lists: 64 tables at a time, two per lane, so that the dependent loads
        // (bounds -> ids) of all tables overlap.  A self-join keeps the query's own row out of the
        // lists and puts it in front: a row of the 10M-row self-join has 91 ids in its 48 lists,
        // 48 of them its own.
        int fill = 0;
        if (SELF) {
            if (lane == 0) buf[0] = q;
            fill = 1;
        }
        for (int t0 = 0; t0 < L; t0 += 64) {
            int s[2], len[2], keep[2];
            uint32_t w[2] = {0, 0};
            int2 be[2] = {make_int2(0, 0), make_int2(0, 0)};
            // neighbouring warps (queries) share the sectors of these table-major reads
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int t = t0 + 32 * h + lane;
                if (t < L) {
                    if (SELF) w[h] = bounds.packed[(size_t)t * n_q + q];
                    else be[h] = bounds.pair[(size_t)t * n_q + q];
                }
            }
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                if (SELF && !(w[h] & PB_PAIR)) be[h] = bounds.unpack(t0 + 32 * h + lane, w[h]);
                s[h] = be[h].x;
                len[h] = be[h].y - be[h].x;
                keep[h] = SELF ? ((w[h] & PB_PAIR) ? 1 : max(len[h] - 1, 0)) : len[h];
            }
            int inc = keep[0] | (keep[1] << 16);  // both prefixes in one scan: at most CAP ids each
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int x = __shfl_up_sync(0xFFFFFFFFu, inc, o);
                if (lane >= o) inc += x;
            }
            const int tot = __shfl_sync(0xFFFFFFFFu, inc, 31);
            const int dst[2] = {fill + (inc & 0xFFFF) - keep[0], fill + (tot & 0xFFFF) + (inc >> 16) - keep[1]};
            int32_t v[2][4];
#pragma unroll
            for (int h = 0; h < 2; ++h)
#pragma unroll
                for (int i = 0; i < 4; ++i) v[h][i] = i < len[h] ? cand[s[h] + i] : 0;
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                if (SELF && (w[h] & PB_PAIR)) buf[dst[h]] = (int32_t)(w[h] & ~PB_PAIR);
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    if (i < len[h]) put_id<SELF>(buf, dst[h] + i, v[h][i], q);
                uint32_t longer = SELF ? __ballot_sync(0xFFFFFFFFu, len[h] > 4) : 0u;
                while (longer) {
                    const int src = __ffs(longer) - 1;
                    longer &= longer - 1;
                    const int ls = __shfl_sync(0xFFFFFFFFu, s[h], src);
                    const int ll = __shfl_sync(0xFFFFFFFFu, len[h], src);
                    const int ld = __shfl_sync(0xFFFFFFFFu, dst[h], src);
                    for (int i = 4 + lane; i < ll; i += 32) put_id<SELF>(buf, ld + i, cand[ls + i], q);
                }
            }
            const int rem[2] = {max(len[0] - 4, 0), max(len[1] - 4, 0)};
            if (!SELF && __any_sync(0xFFFFFFFFu, (rem[0] | rem[1]) != 0)) {
                int ri = rem[0] | (rem[1] << 16);  // at most CAP ids each
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int x = __shfl_up_sync(0xFFFFFFFFu, ri, o);
                    if (lane >= o) ri += x;
                }
                const int rt = __shfl_sync(0xFFFFFFFFu, ri, 31);
                const int pre[2] = {(ri & 0xFFFF) - rem[0], (rt & 0xFFFF) + (ri >> 16) - rem[1]};
                const int n_rem = (rt & 0xFFFF) + (rt >> 16);
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    wl.pre[32 * h + lane] = pre[h];
                    wl.src[32 * h + lane] = s[h] + 4 - pre[h];
                    wl.dst[32 * h + lane] = dst[h] + 4 - pre[h];
                }
                if (lane == 0) wl.pre[64] = n_rem;
                __syncwarp();
                int t = 0;  // the last list that starts at or before a lane's next id
#pragma unroll
                for (int step = 32; step > 0; step >>= 1)
                    if (wl.pre[t + step] <= lane) t += step;
                for (int p0 = lane; p0 - lane < n_rem; p0 += 32 * SM_LOADS) {
                    int32_t x[SM_LOADS];
                    int to[SM_LOADS];
#pragma unroll
                    for (int j = 0; j < SM_LOADS; ++j) {
                        const int p = p0 + 32 * j;
                        x[j] = 0;
                        to[j] = 0;
                        if (p < n_rem) {
                            while (wl.pre[t + 1] <= p) ++t;  // pre[64] = n_rem > p: t stays below 64
                            x[j] = cand[wl.src[t] + p];
                            to[j] = wl.dst[t] + p;
                        }
                    }
#pragma unroll
                    for (int j = 0; j < SM_LOADS; ++j)
                        if (p0 + 32 * j < n_rem) buf[to[j]] = x[j];
                }
                __syncwarp();
            }
            fill += (tot & 0xFFFF) + (tot >> 16);
        }
        __syncwarp();
        int32_t* out = tmp + raw_off[q];
        int written;
        if (r <= 32) written = warp_sort_unique<1>(buf, r, lane, out);
        else if (r <= 64) written = warp_sort_unique<2>(buf, r, lane, out);
        else if (CAP <= 128 || r <= 128) written = warp_sort_unique<4>(buf, r, lane, out);
        else if (r <= 256) written = warp_sort_unique<CAP <= 128 ? 1 : 8>(buf, r, lane, out);
        else if (r <= 512) written = warp_sort_unique<CAP <= 128 ? 1 : 16>(buf, r, lane, out);
        else written = warp_sort_unique<CAP <= 128 ? 1 : 32>(buf, r, lane, out);
        if (lane == 0) uniq_cnt[q] = (uint64_t)written;
        __syncwarp();
    }
}

// ---------------------------------------------------------------------------------------
// Sort path: one CTA per query of mid_list (SMALL_MAX < raw <= MID_MAX), used when the index
// has so many rows that a bitmap would need several windows.  The ids are gathered into
// shared memory, LSD radix sorted there on 8-bit digits (as many passes as the row ids have
// bytes), then adjacent duplicates are dropped while writing out.
// ---------------------------------------------------------------------------------------
constexpr int MS_THREADS = 512;
constexpr int MS_WARPS = MS_THREADS / 32;
constexpr int MS_IPT = 16;
constexpr int MID_MAX = MS_THREADS * MS_IPT;  // 8192

inline size_t sort_path_smem_bytes() {
    return sizeof(uint32_t) * (2 * (size_t)MID_MAX + MS_WARPS * 256 + 256 + 64);
}

__global__ void __launch_bounds__(MS_THREADS)
dedupe_sort_kernel(const uint32_t* __restrict__ mid_list, BoundsView bounds,
                   const int32_t* __restrict__ cand, const uint64_t* __restrict__ raw_off, int L, int id_bytes, int32_t* __restrict__ tmp, uint64_t* __restrict__ uniq_cnt) {
    extern __shared__ __align__(16) uint32_t s_ms[];
    uint32_t* bufA = s_ms;
    uint32_t* bufB = bufA + MID_MAX;
    uint32_t* s_whist = bufB + MID_MAX;       // [MS_WARPS][256]
    uint32_t* s_binstart = s_whist + MS_WARPS * 256;  // [256]
    uint32_t* s_misc = s_binstart + 256;      // [64]
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int q = (int)mid_list[blockIdx.x];
    // gather the bucket lists one after another
    int fill = 0;
    for (int t = 0; t < L; ++t) {
        const int2 be = bounds.get(t, q);
        const int s = be.x, e = be.y;
        for (int i = s + tid; i < e; i += MS_THREADS) bufA[fill + (i - s)] = (uint32_t)cand[i];
        fill += e - s;
    }
    const int r = fill;  // at most MID_MAX: the count that chose this path allows for it
    __syncthreads();
    const int n_iter = (r + MS_THREADS - 1) / MS_THREADS;  // uniform
    uint32_t* src = bufA;
    uint32_t* dst = bufB;
    for (int p = 0; p < id_bytes; ++p) {
        for (int i = tid; i < MS_WARPS * 256; i += MS_THREADS) s_whist[i] = 0;
        __syncthreads();
        uint32_t key[MS_IPT];
        uint16_t rank[MS_IPT];
#pragma unroll
        for (int i = 0; i < MS_IPT; ++i) {
            if (i < n_iter) {
                const int li = warp * (32 * n_iter) + i * 32 + lane;
                const bool valid = li < r;
                key[i] = valid ? src[li] : 0u;
                const uint32_t d = valid ? ((key[i] >> (8 * p)) & 0xFFu) : 0x100u;
                const uint32_t peers = __match_any_sync(0xFFFFFFFFu, d);
                const int leader = __ffs(peers) - 1;
                const uint32_t below = __popc(peers & ((1u << lane) - 1));
                uint32_t old = 0;
                if (valid && lane == leader) old = atomicAdd(&s_whist[warp * 256 + d], (uint32_t)__popc(peers));
                old = __shfl_sync(0xFFFFFFFFu, old, leader);
                rank[i] = (uint16_t)(old + below);
            }
        }
        __syncthreads();
        if (tid < 256) {
            uint32_t cnt = 0;
#pragma unroll
            for (int w = 0; w < MS_WARPS; ++w) {
                uint32_t x = s_whist[w * 256 + tid];
                s_whist[w * 256 + tid] = cnt;
                cnt += x;
            }
            uint32_t inc = cnt;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                uint32_t x = __shfl_up_sync(0xFFFFFFFFu, inc, o);
                if (lane >= o) inc += x;
            }
            if (lane == 31) s_misc[warp] = inc;
            s_binstart[tid] = inc - cnt;  // exclusive inside the warp; warp bases added below
        }
        __syncthreads();
        if (tid < 256) {
            uint32_t wb = 0;
            for (int w = 0; w < warp; ++w) wb += s_misc[w];
            s_binstart[tid] += wb;
        }
        __syncthreads();
#pragma unroll
        for (int i = 0; i < MS_IPT; ++i) {
            if (i < n_iter) {
                const int li = warp * (32 * n_iter) + i * 32 + lane;
                if (li < r) {
                    const uint32_t d = (key[i] >> (8 * p)) & 0xFFu;
                    dst[s_binstart[d] + s_whist[warp * 256 + d] + rank[i]] = key[i];
                }
            }
        }
        __syncthreads();
        uint32_t* tsw = src; src = dst; dst = tsw;
    }
    // adjacent-unique + block compaction, ascending order kept
    int32_t* out = tmp + raw_off[q];
    uint32_t written = 0;  // uniform
    for (int i0 = 0; i0 < r; i0 += MS_THREADS) {
        const int i = i0 + tid;
        bool keep = false;
        uint32_t v = 0;
        if (i < r) {
            v = src[i];
            keep = i == 0 || src[i - 1] != v;
        }
        const uint32_t mask = __ballot_sync(0xFFFFFFFFu, keep);
        if (lane == 0) s_misc[32 + warp] = __popc(mask);
        __syncthreads();
        uint32_t wb = 0, tot = 0;
        for (int w = 0; w < MS_WARPS; ++w) {
            const uint32_t x = s_misc[32 + w];
            if (w < warp) wb += x;
            tot += x;
        }
        if (keep) out[written + wb + __popc(mask & ((1u << lane) - 1))] = (int32_t)v;
        written += tot;
        __syncthreads();
    }
    if (tid == 0) uniq_cnt[q] = (uint64_t)written;
}

// ---------------------------------------------------------------------------------------
// Block path: one CTA per query of big_list.  Row ids are marked in a shared-memory bitmap
// covering a window of `window_bits` ids; windows are visited in increasing order, and as
// every bucket list is ascending each window's slice of a list is found by binary search.
// A pop-count scan of the bitmap then emits the window's ids sorted and unique.
// ---------------------------------------------------------------------------------------
constexpr int BM_THREADS = 1024;
constexpr int BM_WARPS = BM_THREADS / 32;
constexpr int BM_MAX_L = 1024;   // lists kept in shared memory
constexpr int BM_STAGE = 256;    // ids staged per warp before a coalesced flush

__device__ __forceinline__ int lower_bound_i32(const int32_t* __restrict__ a, int lo, int hi, int32_t v) {
    while (lo < hi) {
        int mid = lo + ((hi - lo) >> 1);
        if (a[mid] < v) lo = mid + 1; else hi = mid;
    }
    return lo;
}

inline size_t bitmap_smem_bytes(int window_bits) {
    return (size_t)window_bits / 8 + 3 * BM_MAX_L * sizeof(int) + (size_t)BM_WARPS * BM_STAGE * sizeof(int32_t);
}


// Marks the ids of Lg ascending lists [s_lo[t], s_we[t]) of `cand` in the bitmap.  The lists are
// laid end to end (s_pre = exclusive prefix of their lengths) and that flat sequence is cut
// into equal stretches, one per warp, so the work is balanced however uneven the lists are.
// Must be called by all BM_THREADS threads; s_lo / s_we must be visible (barrier before).
template <int NT = BM_THREADS>
__device__ __forceinline__ void mark_lists_flat(uint32_t* __restrict__ bitmap, const int32_t* __restrict__ cand,
                                                const int* __restrict__ s_lo, const int* __restrict__ s_we,
                                                int* __restrict__ s_pre, uint32_t* __restrict__ s_wtot, int Lg,
                                                int win_lo) {
    constexpr int NWARP = NT / 32;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int len = tid < Lg ? s_we[tid] - s_lo[tid] : 0;
    int inc = len;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        int x = __shfl_up_sync(0xFFFFFFFFu, inc, o);
        if (lane >= o) inc += x;
    }
    if (lane == 31) s_wtot[warp] = (uint32_t)inc;
    __syncthreads();
    int base = 0, total = 0;
    for (int w = 0; w < NWARP; ++w) {
        const int x = (int)s_wtot[w];
        if (w < warp) base += x;
        total += x;
    }
    if (tid < Lg) s_pre[tid] = base + inc - len;
    __syncthreads();
    // Each warp takes a contiguous stretch of the flat sequence; a lane's list index only moves
    // forward (one binary search per warp, then cheap advances), loads stay coalesced and MK of
    // them are in flight per lane.
    constexpr int MK = 20;
    const int per_warp = (((total + NWARP - 1) / NWARP) + 31) & ~31;
    const int w_begin = warp * per_warp, w_end = min(total, w_begin + per_warp);
    if (w_begin < w_end) {
        int t = 0;
        {
            int a = 0, b = Lg - 1;
            while (a < b) {  // largest t with s_pre[t] <= w_begin
                const int mid = (a + b + 1) >> 1;
                if (s_pre[mid] <= w_begin) a = mid; else b = mid - 1;
            }
            t = a;
        }
        for (int e0 = w_begin + lane; e0 - lane < w_end; e0 += 32 * MK) {
            int32_t v[MK];
#pragma unroll
            for (int j = 0; j < MK; ++j) {
                const int e = e0 + 32 * j;
                v[j] = -1;
                if (e < w_end) {
                    while (t + 1 < Lg && s_pre[t + 1] <= e) ++t;
                    v[j] = cand[s_lo[t] + (e - s_pre[t])];
                }
            }
#pragma unroll
            for (int j = 0; j < MK; ++j) {
                if (v[j] >= 0) {
                    const uint32_t id = (uint32_t)(v[j] - win_lo);
                    atomicOr(&bitmap[id >> 5], 1u << (id & 31));
                }
            }
        }
    }
    __syncthreads();
}

__global__ void __launch_bounds__(BM_THREADS)
dedupe_bitmap_kernel(const uint32_t* __restrict__ big_list, BoundsView bounds,
                     const int32_t* __restrict__ cand, const uint64_t* __restrict__ raw_off, int L, int n_rows, int window_bits,
                     int32_t* __restrict__ tmp, uint64_t* __restrict__ uniq_cnt) {
    extern __shared__ __align__(16) uint32_t s_dyn[];
    uint32_t* bitmap = s_dyn;                                       // [window_bits / 32]
    int* s_lo = reinterpret_cast<int*>(bitmap + window_bits / 32);  // [Lc] slice start (global position)
    int* s_hi = s_lo + BM_MAX_L;                                    // [Lc] end of list
    int* s_we = s_hi + BM_MAX_L;                                    // [Lc] end of the window's slice
    int32_t* s_stage = reinterpret_cast<int32_t*>(s_we + BM_MAX_L); // [BM_WARPS][BM_STAGE]
    __shared__ uint32_t s_wtot[BM_WARPS];
    __shared__ int s_any;

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int q = (int)big_list[blockIdx.x];
    const int words = window_bits / 32;
    int32_t* out = tmp + raw_off[q];
    int32_t* stage = s_stage + warp * BM_STAGE;
    uint32_t written = 0;  // uniform across the block

    // L may exceed BM_MAX_L: tables are processed in groups inside the window loop, because
    // every group marks the bitmap of the same window.
    for (int win_lo = 0; win_lo < n_rows; win_lo += window_bits) {
        const int win_hi = min(n_rows, win_lo + window_bits);
        bool cleared = false;
        for (int g0 = 0; g0 < L; g0 += BM_MAX_L) {
            const int Lg = min(BM_MAX_L, L - g0);
            if (tid == 0) s_any = 0;
            __syncthreads();
            for (int t = tid; t < Lg; t += BM_THREADS) {
                const int2 be = bounds.get(g0 + t, q);
                int lo = 0, hi = 0, we = 0;
                if (be.y > be.x) {
                    int s = be.x, e = be.y;
                    if (n_rows <= window_bits) { lo = s; we = e; }
                    else {
                        lo = lower_bound_i32(cand, s, e, win_lo);
                        we = lower_bound_i32(cand, lo, e, win_hi);
                    }
                    hi = e;
                    if (we > lo) s_any = 1;
                }
                s_lo[t] = lo; s_hi[t] = hi; s_we[t] = we;
            }
            __syncthreads();
            const int any = s_any;
            __syncthreads();  // s_any is rewritten at the top of the next group
            if (!any) continue;  // uniform
            if (!cleared) {
                uint4* b4 = reinterpret_cast<uint4*>(bitmap);
                for (int w = tid; w < words / 4; w += BM_THREADS) b4[w] = make_uint4(0, 0, 0, 0);
                cleared = true;
                __syncthreads();
            }
            mark_lists_flat(bitmap, cand, s_lo, s_we, s_hi, s_wtot, Lg, win_lo);
        }
        if (!cleared) continue;  // uniform: nothing in this window
        // ---- pop-count scan.  The window is cut into groups of 128 words (one uint4 per lane);
        // warp w owns groups [w*gpw, (w+1)*gpw). ----
        const uint4* b4 = reinterpret_cast<const uint4*>(bitmap);
        const int groups = words / 128;
        const int gpw = (groups + BM_WARPS - 1) / BM_WARPS;
        const int g_begin = warp * gpw, g_end = min(groups, g_begin + gpw);
        uint32_t wsum = 0;
        for (int g = g_begin; g < g_end; ++g) {
            const uint4 v = b4[g * 32 + lane];
            wsum += __popc(v.x) + __popc(v.y) + __popc(v.z) + __popc(v.w);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) wsum += __shfl_xor_sync(0xFFFFFFFFu, wsum, o);
        if (lane == 0) s_wtot[warp] = wsum;
        __syncthreads();
        uint32_t wbase = 0, wtotal = 0;
        for (int i = 0; i < BM_WARPS; ++i) {
            uint32_t x = s_wtot[i];
            if (i < warp) wbase += x;
            wtotal += x;
        }
        // ---- emit: each lane expands its four words; ids are staged in the warp's slice of
        // shared memory and flushed in coalesced runs; a group denser than the stage is
        // written directly ----
        uint32_t out_pos = written + wbase;  // global position of stage[0]
        uint32_t fill = 0;
        for (int g = g_begin; g < g_end; ++g) {
            const uint4 v = b4[g * 32 + lane];
            const uint32_t wv[4] = {v.x, v.y, v.z, v.w};
            const uint32_t c = __popc(v.x) + __popc(v.y) + __popc(v.z) + __popc(v.w);
            uint32_t inc = c;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                uint32_t x = __shfl_up_sync(0xFFFFFFFFu, inc, o);
                if (lane >= o) inc += x;
            }
            const uint32_t tot = __shfl_sync(0xFFFFFFFFu, inc, 31);
            if (tot == 0) continue;
            const int32_t id0 = win_lo + (g * 128 + lane * 4) * 32;
            if (tot > BM_STAGE || fill + tot > BM_STAGE) {  // flush what is staged
                __syncwarp();
                for (uint32_t i = lane; i < fill; i += 32) out[out_pos + i] = stage[i];
                out_pos += fill;
                fill = 0;
                __syncwarp();
            }
            int32_t* dst = tot > BM_STAGE ? out + out_pos + (inc - c) : stage + fill + (inc - c);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                uint32_t bits = wv[j];
                while (bits) {
                    const int b = __ffs(bits) - 1;
                    bits &= bits - 1;
                    *dst++ = id0 + j * 32 + b;
                }
            }
            if (tot > BM_STAGE) out_pos += tot; else fill += tot;
        }
        __syncwarp();
        for (uint32_t i = lane; i < fill; i += 32) out[out_pos + i] = stage[i];
        written += wtotal;
        __syncthreads();
    }
    if (tid == 0) uniq_cnt[q] = (uint64_t)written;
}

// ---------------------------------------------------------------------------------------
// Window form of the block path: the row range is cut into n_win windows and a CTA takes one
// (query, window) pair.  It
//   1. takes the slices of the query's ascending bucket lists that fall into its window,
//   2. marks their ids in a shared-memory bitmap,
//   3. counts the bits,
//   4. writes the ids of the set bits, ascending, to the place of its slices inside the query's raw span of `tmp` -
//      what is known beforehand, so that no CTA waits for another one.
// compact_windows_kernel brings the pieces together once the counts of all queries are known.
//
// The instructions bound it, not the 8 bytes an id moves (issue slots 89 % taken, the pipe of pop-counts and bit searches 55):
// 10,000 queries of 20,500 entries over a million rows take 823 us and 218 more for the pieces.  Tickets that chained their
// counts and wrote to the final place waited for one another as long as they worked (1,140 us); ids kept in registers,
// ranked by the bits before them and put in order in shared memory have fewer instructions, but random reads of shared
// memory instead, and fewer CTAs fit an SM (890 to 1,400 us).
// ---------------------------------------------------------------------------------------
constexpr int CW_MAX_L = 256;    // lists per query kept in shared memory (<= threads per CTA)

inline size_t window_smem_bytes(int window_bits) {
    return (size_t)window_bits / 8 + (3 * CW_MAX_L + 1) * sizeof(int);  // bitmap, lists
}

// Cuts the ascending lists [s_lo[t], s_we[t]) of `cand` down to their slices in [win_lo, win_hi); an open side of the window
// (the first one's lower, the last one's upper) cuts nothing.  Eight lanes take a (list, side) and look at eight places a step,
// and with two of them in turn a warp has eight searches in flight: what bounds a CTA that has few of them is how many reads wait for
// one another.  Called by all threads, with a barrier before and behind.
template <int NT>
__device__ __forceinline__ void cut_lists(const int32_t* __restrict__ cand, int* __restrict__ s_lo, int* __restrict__ s_we, int L,
                                          int win_lo, int win_hi, bool open_lo, bool open_hi) {
    constexpr int GROUPS = NT / 8;  // a multiple of four: the two sides of a list are in one warp
    const int lane = threadIdx.x & 31, at = threadIdx.x & 7, group = threadIdx.x >> 3, shift = lane & 24;
    for (int p0 = 0; p0 < 2 * L; p0 += 2 * GROUPS) {
        int lo[2], hi[2], target[2];
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const int p = p0 + u * GROUPS + group, t = p >> 1;
            const bool upper = p & 1, have = p < 2 * L;
            lo[u] = have ? s_lo[t] : 0;
            hi[u] = have ? s_we[t] : 0;
            target[u] = upper ? win_hi : win_lo;
            if (!upper && open_lo) hi[u] = lo[u];
            if (upper && open_hi) lo[u] = hi[u];
        }
        while (__any_sync(0xFFFFFFFFu, hi[0] - lo[0] > 8 || hi[1] - lo[1] > 8)) {
            int32_t v[2];
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const int len = hi[u] - lo[u];
                v[u] = len > 8 ? cand[lo[u] + (at + 1) * (len / 9)] : 0;
            }
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const int len = hi[u] - lo[u], step = len / 9;
                const int c = __popc((__ballot_sync(0xFFFFFFFFu, len > 8 && v[u] < target[u]) >> shift) & 0xFFu);  // lanes 0 .. c - 1
                if (len > 8) {
                    if (c < 8) hi[u] = lo[u] + (c + 1) * step;
                    if (c > 0) lo[u] += c * step + 1;
                }
            }
        }
        int32_t v[2];
#pragma unroll
        for (int u = 0; u < 2; ++u) v[u] = at < hi[u] - lo[u] ? cand[lo[u] + at] : 0;
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const int c = __popc((__ballot_sync(0xFFFFFFFFu, at < hi[u] - lo[u] && v[u] < target[u]) >> shift) & 0xFFu);
            const int p = p0 + u * GROUPS + group;
            if (at == 0 && p < 2 * L) ((p & 1) ? s_we : s_lo)[p >> 1] = lo[u] + c;
        }
        __syncwarp();
    }
}

// Walk over the Lg lists [s_lo[t], s_lo[t] + len_t) laid end to end (s_pre[t] = exclusive prefix
// of the lengths, s_pre[Lg] = total).  The flat sequence is cut into equal stretches, one per warp;
// a batch is 32 * MK consecutive elements of the stretch: lanes read consecutive elements
// (coalesced) and every lane has MK independent loads in flight.  The loaded ids are handed back
// untouched (-1 past the end) so that the caller decides when to consume them.
template <int NT, int MK>
struct ListWalk {
    int t, next, base, w_begin, w_end, per_warp;

    __device__ __forceinline__ void init(const int* __restrict__ s_lo, const int* __restrict__ s_pre, int Lg) {
        constexpr int NWARP = NT / 32;
        const int warp = threadIdx.x >> 5;
        const int total = s_pre[Lg];
        per_warp = (((total + NWARP - 1) / NWARP) + 31) & ~31;
        w_begin = warp * per_warp;
        w_end = min(total, w_begin + per_warp);
        t = 0; next = 0; base = 0;
        if (w_begin < w_end) {
            int a = 0, b = Lg - 1;
            while (a < b) {  // largest t with s_pre[t] <= w_begin
                const int mid = (a + b + 1) >> 1;
                if (s_pre[mid] <= w_begin) a = mid; else b = mid - 1;
            }
            t = a;
            next = s_pre[t + 1];        // first flat position past list t
            base = s_lo[t] - s_pre[t];  // flat position -> position in cand
        }
    }
    // batch whose first element (of lane 0) is the flat position e0 - lane
    __device__ __forceinline__ void load(const int32_t* __restrict__ cand, const int* __restrict__ s_lo,
                                         const int* __restrict__ s_pre, int e0, int32_t (&v)[MK]) {
#pragma unroll
        for (int j = 0; j < MK; ++j) {
            const int e = e0 + 32 * j;
            v[j] = -1;
            if (e < w_end) {
                while (e >= next) {  // e < total, so t stays below Lg
                    ++t;
                    next = s_pre[t + 1];
                    base = s_lo[t] - s_pre[t];
                }
                v[j] = cand[base + e];
            }
        }
    }
};

// Slice of every bucket list that falls into every window: slices[(b * n_win + w) * L + t] =
// [a, z) in cand for the query big_list[b].  One thread per (query, list, window) finds the window's lower boundary with a
// binary search and writes it as the start of its own slice and the end of the previous one;
// with a million independent searches in flight the dependent loads cost nothing, whereas
// inside the window kernel they would sit on the critical path of every CTA.
__global__ void __launch_bounds__(256)
slice_lists_kernel(const uint32_t* __restrict__ big_list, BoundsView bounds, const int32_t* __restrict__ cand, int n_big, int L,
                   int window_bits, int n_win, int2* __restrict__ slices, KernelBefore kernel_before) {
    behind_kernel_before(big_list, cand, slices, kernel_before);
    const size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= (size_t)n_big * L * n_win) return;
    const int w = (int)(idx % n_win);
    const size_t pair = idx / n_win;  // b * L + t
    const int b = (int)(pair / L), t = (int)(pair - (size_t)b * L);
    const int2 be = bounds.get(t, (int)big_list[b]);
    const int lo = be.x, we = be.y;
    int* flat = reinterpret_cast<int*>(slices);
    const size_t mine = (((size_t)b * n_win + w) * L + t) * 2;
    int a = lo;
    if (w > 0) {
        const long long bound = (long long)w * window_bits;
        a = bound > 0x7FFFFFFFll ? we : lower_bound_i32(cand, lo, we, (int32_t)bound);
        flat[mine - (size_t)L * 2 + 1] = a;  // end of the previous window's slice
    }
    flat[mine] = a;
    if (w == n_win - 1) flat[mine + 1] = we;
}

// pieces[b * n_win + w]: x = where the piece starts inside the query's raw span, y = its ids.  A launch whose counts the
// host has not seen covers all queries: n_big says how many there are to do, and `room` is as in dedupe_small_kernel.
template <int NT, int MK>
__global__ void __launch_bounds__(NT, 1920 / NT)  // cut_lists would take it to 37 registers and to four CTAs of 384 threads an SM
dedupe_window_kernel(const uint32_t* __restrict__ big_list, BoundsView bounds, const int32_t* __restrict__ cand,
                     const uint64_t* __restrict__ raw_off, int L, int n_rows, int window_bits, int n_win, bool self_join,
                     const int2* __restrict__ slices /* or null */, const uint32_t* __restrict__ n_big /* or null: all */, uint64_t room,
                     int32_t* __restrict__ tmp, uint2* __restrict__ pieces, unsigned long long* __restrict__ uniq_cnt, KernelBefore kernel_before) {
    behind_kernel_before(big_list, cand, raw_off, slices, n_big, tmp, pieces, uniq_cnt, kernel_before);
    constexpr int NWARP = NT / 32;
    extern __shared__ __align__(16) uint32_t s_dyn[];
    const int n32 = window_bits / 32;                        // a multiple of 128
    uint32_t* bm32 = s_dyn;                                  // [n32] bitmap
    int* s_lo = reinterpret_cast<int*>(bm32 + n32);          // [L] slice start in cand
    int* s_we = s_lo + CW_MAX_L;                             // [L] slice end
    int* s_pre = s_we + CW_MAX_L;                            // [L + 1] prefix of slice lengths
    __shared__ uint32_t s_wtot[NWARP];
    __shared__ uint32_t s_wskip[NWARP];

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int slot = blockIdx.x / n_win, w = blockIdx.x - slot * n_win;
    if (n_big && (slot >= (int)*n_big || raw_off[bounds.n_q] > room)) return;
    const int q = (int)big_list[slot];
    const int win_lo = w * window_bits;
    const int win_hi = min(n_rows, win_lo + window_bits);
    // ---- 1. clear, slices, their prefix and the raw ids of the windows before this one ----
    int first = 0;  // of this thread's whole list
    int2 mine = make_int2(0, 0);
    if (slices) {
        if (tid < L) {
            mine = slices[(size_t)blockIdx.x * L + tid];
            first = slices[(size_t)slot * n_win * L + tid].x;
        }
    } else if (tid < L) {
        mine = bounds.get(tid, q);
        first = mine.x;
    }
    {
        uint4* b4 = reinterpret_cast<uint4*>(bm32);
        for (int i = tid; i < n32 / 4; i += NT) b4[i] = make_uint4(0, 0, 0, 0);
    }
    if (!slices && n_win > 1) {
        if (tid < L) { s_lo[tid] = mine.x; s_we[tid] = mine.y; }
        __syncthreads();
        cut_lists<NT>(cand, s_lo, s_we, L, win_lo, win_hi, w == 0, w == n_win - 1);
        __syncthreads();
        if (tid < L) mine = make_int2(s_lo[tid], s_we[tid]);
    }
    // A self-join's raw count takes the own row off every list and adds it once, and so does the place of a piece:
    // a list with ids before this window has the own row among them if that lies there.
    const bool own_before = self_join && q < win_lo;
    uint32_t skip = (uint32_t)(mine.x - first);
    if (own_before && skip) --skip;
    {   // exclusive prefix of the slice lengths (L <= NT)
        const int len = mine.y - mine.x;
        int inc = len;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int x = __shfl_up_sync(0xFFFFFFFFu, inc, o);
            if (lane >= o) inc += x;
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) skip += __shfl_xor_sync(0xFFFFFFFFu, skip, o);
        if (lane == 31) { s_wtot[warp] = (uint32_t)inc; s_wskip[warp] = skip; }
        if (tid < L) s_lo[tid] = mine.x;
        __syncthreads();
        int base = 0;
        for (int i = 0; i < warp; ++i) base += (int)s_wtot[i];
        if (tid < L) s_pre[tid] = base + inc - len;
        if (tid == L - 1) s_pre[L] = base + inc;
        skip = own_before ? 1u : 0u;
        for (int i = 0; i < (L + 31) / 32; ++i) skip += s_wskip[i];
    }
    __syncthreads();
    // ---- 2. mark ----
    {
        ListWalk<NT, MK> wk;
        wk.init(s_lo, s_pre, L);
        int32_t v[MK];
        for (int e0 = wk.w_begin + lane; e0 - lane < wk.w_end; e0 += 32 * MK) {
            wk.load(cand, s_lo, s_pre, e0, v);
#pragma unroll
            for (int j = 0; j < MK; ++j) {
                if (v[j] >= 0) {
                    const uint32_t id = (uint32_t)(v[j] - win_lo);
                    atomicOr(&bm32[id >> 5], 1u << (id & 31));
                }
            }
        }
    }
    __syncthreads();
    // ---- 3. count.  The bitmap in groups of 128 words, one uint4 a lane; a warp owns a stretch of groups. ----
    const uint4* bm4 = reinterpret_cast<const uint4*>(bm32);
    const int groups = n32 / 128, per_warp = (groups + NWARP - 1) / NWARP;
    const int g_begin = min(groups, warp * per_warp), g_end = min(groups, g_begin + per_warp);
    uint32_t sum = 0;
    for (int g = g_begin; g < g_end; ++g) {
        const uint4 x = bm4[g * 32 + lane];
        sum += __popc(x.x) + __popc(x.y) + __popc(x.z) + __popc(x.w);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xFFFFFFFFu, sum, o);
    if (lane == 0) s_wtot[warp] = sum;
    __syncthreads();
    uint32_t at = 0, total = 0;
    for (int i = 0; i < NWARP; ++i) {
        const uint32_t x = s_wtot[i];
        if (i < warp) at += x;
        total += x;
    }
    if (tid == 0) {
        pieces[blockIdx.x] = make_uint2(skip, total);
        if (n_win == 1) uniq_cnt[q] = total;
        else if (total) atomicAdd(&uniq_cnt[q], (unsigned long long)total);
    }
    // ---- 4. emit.  Most words have an id or none: the first goes without a loop (10,000 sets of 18,500 ids of a million rows: the whole case 2,331 ->
    // 2,298 us; with two or three without one 2,296 and 2,317, and sparser sets slower). ----
    int32_t* out = tmp + raw_off[q] + skip + at;
    for (int g = g_begin; g < g_end; ++g) {
        const uint4 x = bm4[g * 32 + lane];
        const uint32_t wv[4] = {x.x, x.y, x.z, x.w};
        const uint32_t c = __popc(x.x) + __popc(x.y) + __popc(x.z) + __popc(x.w);
        uint32_t inc = c;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, inc, o);
            if (lane >= o) inc += y;
        }
        int32_t* dst = out + (inc - c);
        const int32_t id0 = win_lo + (g * 128 + lane * 4) * 32;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            uint32_t bits = wv[j];
            int32_t* const end = dst + __popc(bits);
            if (bits) *dst = id0 + j * 32 + (__ffs(bits) - 1);
            for (bits &= bits - 1; bits; bits &= bits - 1) *++dst = id0 + j * 32 + (__ffs(bits) - 1);
            dst = end;
        }
        out += __shfl_sync(0xFFFFFFFFu, inc, 31);
    }
}

// ---------------------------------------------------------------------------------------
// Compaction of the per-query segments from their raw offsets to their final offsets.
// ---------------------------------------------------------------------------------------
// Queries of big_list in [q_lo, q_hi): a whole block copies the segment, to out[offsets[q] - first ...].
__global__ void __launch_bounds__(256)
compact_big_kernel(const uint32_t* __restrict__ big_list, const int32_t* __restrict__ tmp,
                   const uint64_t* __restrict__ raw_off, const uint64_t* __restrict__ uniq_cnt,
                   const uint64_t* __restrict__ offsets, uint32_t q_lo, uint32_t q_hi, uint64_t first, int32_t* __restrict__ out) {
    const uint32_t q = big_list[blockIdx.x];
    if (q < q_lo || q >= q_hi) return;
    const uint64_t c = uniq_cnt[q];
    const int32_t* src = tmp + raw_off[q];
    int32_t* dst = out + (offsets[q] - first);
    for (uint64_t i = threadIdx.x; i < c; i += blockDim.x) dst[i] = src[i];
}

// The pieces of the queries that went through dedupe_window_kernel, a CTA per (query, window): queries [q_lo, q_hi), to
// out[offsets[q] - first ...].  Bound by the 8 bytes an id moves.
constexpr int CWN_LOADS = 8;
__global__ void __launch_bounds__(256)
compact_windows_kernel(const uint32_t* __restrict__ big_list, const int32_t* __restrict__ tmp, const uint64_t* __restrict__ raw_off,
                       const uint2* __restrict__ pieces, const uint64_t* __restrict__ offsets, int n_win, uint32_t q_lo, uint32_t q_hi,
                       uint64_t first, int32_t* __restrict__ out, KernelBefore kernel_before) {
    behind_kernel_before(big_list, tmp, raw_off, pieces, offsets, out, kernel_before);
    const int slot = blockIdx.x / n_win, w = blockIdx.x - slot * n_win;
    const uint32_t q = big_list[slot];
    if (q < q_lo || q >= q_hi) return;
    uint32_t before = 0;  // ids of the pieces before this one: at most as many as rows
    for (int i = threadIdx.x & 31; i < w; i += 32) before += pieces[slot * (size_t)n_win + i].y;
    const uint64_t to = offsets[q] - first + __reduce_add_sync(0xFFFFFFFFu, before);
    const uint2 p = pieces[blockIdx.x];
    const int32_t* src = tmp + raw_off[q] + p.x;
    int32_t* dst = out + to;
    for (uint32_t i0 = threadIdx.x; i0 < p.y; i0 += 256 * CWN_LOADS) {
        int32_t v[CWN_LOADS];
#pragma unroll
        for (int j = 0; j < CWN_LOADS; ++j) v[j] = i0 + 256 * j < p.y ? src[i0 + 256 * j] : 0;
#pragma unroll
        for (int j = 0; j < CWN_LOADS; ++j)
            if (i0 + 256 * j < p.y) dst[i0 + 256 * j] = v[j];
    }
}

// Small queries only (big ones are copied by the two kernels above).  A warp takes `per` <= 32 queries
// (few for a small set, which would leave the chip idle otherwise), reads
// their descriptors with one coalesced load each and copies CS_ROWS segments at a time, two words
// per lane each, so that 2 * CS_ROWS independent loads are in flight; one segment after another
// left the copy of the 10M-row self-join's 1.8 GB at 1.6 TB/s.
constexpr int CS_ROWS = 4;
__global__ void __launch_bounds__(256)
compact_small_kernel(const int32_t* __restrict__ tmp, const uint64_t* __restrict__ raw_cnt,
                     const uint64_t* __restrict__ raw_off, const uint64_t* __restrict__ uniq_cnt,
                     const uint64_t* __restrict__ offsets, int n_q, int per, uint64_t first, int32_t* __restrict__ out, KernelBefore kernel_before) {
    behind_kernel_before(tmp, raw_cnt, raw_off, uniq_cnt, offsets, out, kernel_before);
    const int lane = threadIdx.x & 31;
    const size_t warp = ((size_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const size_t n_warps = ((size_t)gridDim.x * blockDim.x) >> 5;
    for (size_t q0 = warp * per; q0 < (size_t)n_q; q0 += n_warps * per) {
        const size_t q = q0 + lane;
        uint64_t from = 0, to = 0;
        int cnt = 0;
        if (lane < per && q < (size_t)n_q && raw_cnt[q] <= SMALL_MAX) {
            cnt = (int)uniq_cnt[q];
            from = raw_off[q];
            to = offsets[q] - first;
        }
        for (int i = 0; i < per; i += CS_ROWS) {
            const int32_t* src[CS_ROWS];
            int32_t* dst[CS_ROWS];
            int c[CS_ROWS], most = 0;
#pragma unroll
            for (int j = 0; j < CS_ROWS; ++j) {
                src[j] = tmp + __shfl_sync(0xFFFFFFFFu, from, i + j);
                dst[j] = out + __shfl_sync(0xFFFFFFFFu, to, i + j);
                c[j] = __shfl_sync(0xFFFFFFFFu, cnt, i + j);
                most = max(most, c[j]);
            }
            for (int e = lane; e - lane < most; e += 64) {
                int32_t a[CS_ROWS], b[CS_ROWS];
#pragma unroll
                for (int j = 0; j < CS_ROWS; ++j) {
                    a[j] = e < c[j] ? src[j][e] : 0;
                    b[j] = e + 32 < c[j] ? src[j][e + 32] : 0;
                }
#pragma unroll
                for (int j = 0; j < CS_ROWS; ++j) {
                    if (e < c[j]) dst[j][e] = a[j];
                    if (e + 32 < c[j]) dst[j][e + 32] = b[j];
                }
            }
        }
    }
}

// ---------------------------------------------------------------------------------------
// Batch / shard merging helpers.
// ---------------------------------------------------------------------------------------
// offsets_out[q0 + i] = offsets_in[i] + shift, i in [0, n]
__global__ void shift_offsets_kernel(const uint64_t* __restrict__ in, size_t n, uint64_t shift,
                                     uint64_t* __restrict__ out) {
    size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = in[i] + shift;
}

// counts[q] = sum over shards of (off_r[q+1] - off_r[q])
__global__ void shard_counts_kernel(const uint64_t* const* __restrict__ shard_offsets, int n_shards,
                                    int n_q, uint64_t* __restrict__ counts) {
    int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= n_q) return;
    uint64_t c = 0;
    for (int r = 0; r < n_shards; ++r) c += shard_offsets[r][q + 1] - shard_offsets[r][q];
    counts[q] = c;
}

// One CTA per query (grid-stride): the shards' lists, shifted to global ids, in shard order.  The
// shard buffers may be peer memory, so the per-shard offsets of a query are fetched by one thread
// each (one round trip instead of one per shard), and the lists are copied as one flat sequence
// with eight independent loads in flight per thread to cover the link latency.
constexpr int SI_GROUP = 64;   // shards handled per sweep
constexpr int SI_UNROLL = 8;
__global__ void __launch_bounds__(256)
shard_interleave_kernel(const int32_t* const* __restrict__ shard_indices,
                        const uint64_t* const* __restrict__ shard_offsets,
                        const int64_t* __restrict__ row_base, int n_shards, int n_q,
                        const uint64_t* __restrict__ offsets, int32_t* __restrict__ out) {
    __shared__ const int32_t* s_src[SI_GROUP];   // shard list of this query, already at its start
    __shared__ uint64_t s_pre[SI_GROUP + 1];     // exclusive prefix of the list lengths
    __shared__ int32_t s_base[SI_GROUP];
    const int tid = threadIdx.x;
    for (size_t q = blockIdx.x; q < (size_t)n_q; q += gridDim.x) {
        uint64_t o = offsets[q];
        for (int g0 = 0; g0 < n_shards; g0 += SI_GROUP) {
            const int G = min(SI_GROUP, n_shards - g0);
            __syncthreads();  // the previous sweep is done with the tables
            if (tid < G) {
                const uint64_t* po = shard_offsets[g0 + tid];
                const uint64_t s = po[q], e = po[q + 1];
                s_src[tid] = shard_indices[g0 + tid] + s;
                s_pre[tid + 1] = e - s;  // length for now
                s_base[tid] = (int32_t)row_base[g0 + tid];
            }
            __syncthreads();
            if (tid == 0) {
                uint64_t run = 0;
                for (int r = 0; r < G; ++r) {
                    const uint64_t len = s_pre[r + 1];
                    s_pre[r] = run;
                    run += len;
                }
                s_pre[G] = run;
            }
            __syncthreads();
            const uint64_t total = s_pre[G];
            int r = 0;
            for (uint64_t i0 = tid; i0 < total; i0 += 256 * SI_UNROLL) {
                // the loaded value is not touched before all loads are issued: an add right after
                // the load would make every load wait for the one before it
                int32_t v[SI_UNROLL], shift[SI_UNROLL];
#pragma unroll
                for (int j = 0; j < SI_UNROLL; ++j) {
                    const uint64_t i = i0 + 256 * j;
                    v[j] = 0;
                    shift[j] = 0;
                    if (i < total) {
                        while (i >= s_pre[r + 1]) ++r;  // i < total keeps r below G
                        shift[j] = s_base[r];
                        v[j] = s_src[r][i - s_pre[r]];
                    }
                }
#pragma unroll
                for (int j = 0; j < SI_UNROLL; ++j) {
                    const uint64_t i = i0 + 256 * j;
                    if (i < total) out[o + i] = v[j] + shift[j];
                }
            }
            o += total;
        }
    }
}

// one warp per query, for results with short lists
__global__ void __launch_bounds__(256)
shard_interleave_small_kernel(const int32_t* const* __restrict__ shard_indices,
                              const uint64_t* const* __restrict__ shard_offsets,
                              const int64_t* __restrict__ row_base, int n_shards, int n_q,
                              const uint64_t* __restrict__ offsets, int32_t* __restrict__ out) {
    const int lane = threadIdx.x & 31;
    const size_t warp = ((size_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const size_t n_warps = ((size_t)gridDim.x * blockDim.x) >> 5;
    for (size_t q = warp; q < (size_t)n_q; q += n_warps) {
        uint64_t o = offsets[q];
        for (int r = 0; r < n_shards; ++r) {
            const uint64_t s = shard_offsets[r][q], e = shard_offsets[r][q + 1];
            const int32_t* src = shard_indices[r] + s;
            const int32_t base = (int32_t)row_base[r];
            for (uint64_t i = lane; i < e - s; i += 32) out[o + i] = src[i] + base;
            o += e - s;
        }
    }
}

// ---------------------------------------------------------------------------------------
// Push form of the shard exchange.  Every rank holds the per-query unique counts of all ranks
// (counts_all[r][q]); rank `rank` needs, for each query, where its own list starts inside the
// merged list held by the query's owner (owner = q / per: the ranks own equal slices of the
// queries), and the owner needs the counts / offsets of its slice.
// ---------------------------------------------------------------------------------------
// merged[q] = sum over ranks of counts_all[r][q]; before_me[q] = the part of it from ranks below `rank`
__global__ void __launch_bounds__(256)
exchange_counts_kernel(const uint64_t* __restrict__ counts_all, int n_ranks, int rank, int n_q,
                       uint64_t* __restrict__ merged, uint64_t* __restrict__ before_me) {
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= n_q) return;
    uint64_t all = 0, below = 0;
    for (int r = 0; r < n_ranks; ++r) {
        const uint64_t c = counts_all[(size_t)r * n_q + q];
        if (r < rank) below += c;
        all += c;
    }
    merged[q] = all;
    before_me[q] = below;
}

// S = exclusive scan of merged over all queries (n_q + 1 entries).  dstpos[q] = position of this
// rank's list of query q inside the owner's merged id array; the owner's own slice [my_lo, my_hi)
// gets its counts and offsets; slice_totals[j] = ids of slice j.
__global__ void __launch_bounds__(256)
exchange_positions_kernel(const uint64_t* __restrict__ S, const uint64_t* __restrict__ merged,
                          const uint64_t* __restrict__ before_me, int n_q, int per, int n_ranks, int my_lo,
                          int my_hi, uint64_t* __restrict__ dstpos, uint64_t* __restrict__ my_counts,
                          uint64_t* __restrict__ my_offsets, uint64_t* __restrict__ slice_totals) {
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q < n_ranks) {
        const int lo = min(n_q, q * per), hi = min(n_q, lo + per);
        slice_totals[q] = S[hi] - S[lo];
    }
    if (q > n_q) return;
    if (q < n_q) dstpos[q] = S[q] - S[min(n_q, (q / per) * per)] + before_me[q];
    if (q >= my_lo && q <= my_hi) {
        my_offsets[q - my_lo] = S[q] - S[my_lo];
        if (q < my_hi) my_counts[q - my_lo] = merged[q];
    }
}

// This rank's lists, shifted to global row ids, stored into the owners' id arrays (recv[j] may
// be peer memory: plain coalesced stores, reads are local).  Queries are visited in an order
// that deals the owners round-robin, shifted by the rank: step v goes to owner (v + rank) mod
// n_ranks.  In query order every rank would store to owner 0 first, then to owner 1 ... - all
// ranks into one GPU's NVLink ingress while the other links idle (measured at 8 GPUs: push +
// wait for the slowest rank 3.3 ms for 642 MB per GPU, four times the link time).
__device__ __forceinline__ long long exchange_query_of_step(size_t v, int n_ranks, int rank, int per, int n_q) {
    const int owner = (int)((v + (size_t)rank) % (size_t)n_ranks);
    const long long q = (long long)owner * per + (long long)(v / (size_t)n_ranks);
    return q < (long long)n_q ? q : -1;
}

// CTA per query for long lists.  The stores are 16 bytes per thread on 16-byte boundaries of the
// destination (a warp writes 512 contiguous bytes: whole NVLink packets whatever the phase of the
// list inside the owner's array); the few ids before the first boundary and after the last one
// go out one by one.  The local reads are plain 4-byte loads, sixteen in flight per thread.
constexpr int SP_UNROLL = 4;

__global__ void __launch_bounds__(256)
shard_push_kernel(const int32_t* __restrict__ idx, const uint64_t* __restrict__ off,
                  const uint64_t* __restrict__ dstpos, int32_t* const* __restrict__ recv, int per, int n_q,
                  int n_ranks, int rank, int32_t row_base) {
    const size_t n_steps = (size_t)per * n_ranks;
    for (size_t v = blockIdx.x; v < n_steps; v += gridDim.x) {
        const long long q = exchange_query_of_step(v, n_ranks, rank, per, n_q);
        if (q < 0) continue;
        const uint64_t s = off[q], len = off[q + 1] - s;
        if (len == 0) continue;
        const int32_t* src = idx + s;
        int32_t* dst = recv[q / per] + dstpos[q];
        const uint64_t head = min(len, (uint64_t)(((16u - (uint32_t)(reinterpret_cast<uintptr_t>(dst) & 15u)) & 15u) >> 2));
        if (threadIdx.x < head) dst[threadIdx.x] = src[threadIdx.x] + row_base;
        const uint64_t n4 = (len - head) >> 2;
        const int32_t* s2 = src + head;
        int4* d4 = reinterpret_cast<int4*>(dst + head);
        for (uint64_t i0 = threadIdx.x; i0 < n4; i0 += 256 * SP_UNROLL) {
            int4 w[SP_UNROLL];
#pragma unroll
            for (int j = 0; j < SP_UNROLL; ++j) {
                const uint64_t i = i0 + 256 * j;
                if (i < n4) {
                    const int32_t* p = s2 + 4 * i;
                    w[j] = make_int4(p[0], p[1], p[2], p[3]);
                }
            }
#pragma unroll
            for (int j = 0; j < SP_UNROLL; ++j) {
                const uint64_t i = i0 + 256 * j;
                if (i < n4)
                    d4[i] = make_int4(w[j].x + row_base, w[j].y + row_base, w[j].z + row_base, w[j].w + row_base);
            }
        }
        const uint64_t done = head + 4 * n4;
        if (done + threadIdx.x < len) dst[done + threadIdx.x] = src[done + threadIdx.x] + row_base;
    }
}

// warp per query, for results with short lists
__global__ void __launch_bounds__(256)
shard_push_small_kernel(const int32_t* __restrict__ idx, const uint64_t* __restrict__ off,
                        const uint64_t* __restrict__ dstpos, int32_t* const* __restrict__ recv, int per,
                        int n_q, int n_ranks, int rank, int32_t row_base) {
    const int lane = threadIdx.x & 31;
    const size_t warp = ((size_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const size_t n_warps = ((size_t)gridDim.x * blockDim.x) >> 5;
    const size_t n_steps = (size_t)per * n_ranks;
    for (size_t v = warp; v < n_steps; v += n_warps) {
        const long long q = exchange_query_of_step(v, n_ranks, rank, per, n_q);
        if (q < 0) continue;
        const uint64_t s = off[q], len = off[q + 1] - s;
        int32_t* dst = recv[q / per] + dstpos[q];
        for (uint64_t i = lane; i < len; i += 32) dst[i] = idx[s + i] + row_base;
    }
}

}  // namespace culsh_b200
