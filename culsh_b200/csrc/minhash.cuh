// MinHash signatures over CSR rows.  Replaces compute_minhash_kernel
// (minhash/hash.cuh:69-128): sig[t][row][j] = min over the row's column ids c of
// (A[h]*c + B[h]) mod 4294967291, h = t*k + j; an empty row gives 0xFFFFFFFF.
//
// One warp per row.  Lanes own hash functions (lane, lane+32, ...), so every lane is busy
// however short the row is and no cross-lane reduction is needed; the row's column ids
// are loaded 32 at a time (coalesced) and reach all lanes through shared memory or shuffles.  The modulus is
// folded with 2^32 = 5 (mod p) instead of a 64-bit division.
#pragma once

#include "common.cuh"

namespace culsh_b200 {

constexpr uint32_t MINHASH_PRIME = 4294967291u;  // minhash/hash.cuh:17
constexpr int MH_STEPS = 4;  // pairs of ids a turn of the loop
// A warp is a CTA of its own: rows differ in length tenfold, and with eight warps a CTA held its place until the longest of their
// rows was over.  Its rows lie next to one another: their bounds are one load, the ids of the next row follow those of this one,
// and a line of ids or of keys has one user.  With rows a grid apart a row waited for its bounds and then for its ids, which short
// rows do not cover (2M rows of 5 ids below 2^16 into 32 functions 541 us, 394 this way; eight warps a CTA, with twice the warps an SM,
// 438.  2M of 20 to 200 ids into 128 with 10,000 queries 4,450 and 4,244).
constexpr int MH_THREADS = 32;
// Rows of a warp, at most (fewer than 32: a lane each for their bounds): many for what it sets up once, few for the last warps to
// end together, but no fewer warps than MH_WARPS of an SM, eight turns (with rows a grid apart, 2M sets: 4 rows 4,525 us, 16
// 4,450, 64 4,497; 100,003: 4 rows 248, 16 269, 64 288).
constexpr int MH_ROWS = 16;
constexpr int MH_WARPS = 192;
constexpr int MH_MAX_PER_LANE = 8;               // hashes per lane per sweep (H <= 256 in one sweep)

__device__ __forceinline__ uint64_t mad_wide_u32(uint32_t a, uint32_t b, uint64_t c) {
    uint64_t d;
    asm("mad.wide.u32 %0, %1, %2, %3;" : "=l"(d) : "r"(a), "r"(b), "l"(c));
    return d;
}

// (a*c + b) mod p with p = 2^32 - 5, i.e. 2^32 == 5 (mod p), for a, b < p and c < 2^31.
// x = a*c + b < 2^63; y = 5*x_hi + x_lo < 3.5 * 2^32 is congruent to x; s = 5*y_hi + y_lo
// < 2^32 + 15 is congruent too and lies below 2p, so the result is s or s - p.  s >= p exactly
// when s + 5 carries out of 32 bits, and then (s + 5) mod 2^32 = s - p: one add with a carry
// test replaces the compare-and-subtract.  b64 is b zero-extended (the caller keeps it in
// registers across the row).
__device__ __forceinline__ uint32_t hash_mod_prime(uint32_t a, uint32_t c, uint64_t b64) {
    const uint64_t x = mad_wide_u32(a, c, b64);
    const uint64_t y = mad_wide_u32((uint32_t)(x >> 32), 5u, (uint64_t)(uint32_t)x);
    const uint32_t u = 5u * (uint32_t)(y >> 32) + 5u;   // <= 20
    const uint32_t t = (uint32_t)y + u;                 // (s + 5) mod 2^32
    return t < u ? t : t - 5u;                          // carried: s - p; else s
}

// Row loop form: the value shifted by 5, without the final correction.  x = a*c + b5 with b5 = b + 5
// is folded until the last fold t wraps at most once; a wrap is worth another 5 (2^32 == 5) and
// cannot wrap again.  The result is congruent to value + 5 and below 2^32: value + 5
// itself, except that value + 5 >= p may come out as value + 5 - p, which is below 5 and nothing else
// is.  A (row, hash function) whose minimum ends up there (5 in 2^32 per evaluation) is evaluated again in
// full.  For c < 2^29 5*x_hi fits 32 bits and one 32-bit fold does.  The multiply pipe bounds the
// kernel and a wide multiply-add takes two of its slots: with two wide folds and a wrap flag kept
// per evaluation 2M sets of 110 ids x 128 functions took 11.0 ms, with this form 7.75.
constexpr uint32_t MH_FAST_COL = 1u << 29;
__device__ __forceinline__ uint32_t hash_plus5(uint32_t a, uint32_t c, uint64_t b5) {
    const uint64_t x = mad_wide_u32(a, c, b5);
    const uint32_t lo = (uint32_t)x, t = lo + 5u * (uint32_t)(x >> 32);
    return t < lo ? t + 5u : t;
}
__device__ __forceinline__ uint32_t hash_plus5_any(uint32_t a, uint32_t c, uint64_t b5) {
    const uint64_t x = mad_wide_u32(a, c, b5);
    const uint64_t y = mad_wide_u32((uint32_t)(x >> 32), 5u, (uint64_t)(uint32_t)x);
    const uint32_t lo = (uint32_t)y, t = lo + 5u * (uint32_t)(y >> 32);
    return t < lo ? t + 5u : t;
}

// Column ids below 2^20: a*c + b5 + 2^52 is below 2^53, so that one double-precision multiply-add gives it exactly, the low
// word of x in the low word of the result and the high word of x behind the constant exponent in the other.  The double
// pipe, which nothing else here uses, takes a warp's multiply-add in two cycles, the integer one a wide one in eight.  What
// is left is bound by issue.
//
// Ids below 2^16 leave the wrap of the fold out, which takes the evaluation to three instructions (the multiply-add, the fold,
// an add with the minimum in one): x_hi is at most the id + 1, so a fold that wraps comes out below MH_AGAIN, and a
// minimum at or above that is right.  One below it, rare as long as the row is short (about 8e-5 for each id), is evaluated again in
// full by the whole warp.  A step of 32 ids is sorted into those below and above through shared memory, as the doubles that
// all lanes then read.  2M sets of 20 to 200 ids into 128 hash functions (with the 10,000 queries): 7,730 us in the integer form,
// 6,630 with the wrap for all, 4,870 without (two pairs of ids a turn 4,900, the line at 2^14 4,940); 100,003 sets 414, 367 and 278.
constexpr uint32_t MH_DOUBLE_COL = 1u << 20;
constexpr double MH_2_52 = 4503599627370496.0;
constexpr uint32_t MH_2_52_HI = 0x43300000u;
constexpr uint32_t MH_SHORT_COL = 1u << 16;
constexpr uint32_t MH_AGAIN = 5u * (MH_SHORT_COL + 1u);
constexpr int MH_SHORT_ROW = 1024;  // ids of a row: at the line a twelfth of the minima is evaluated again
// b52 = b + 5 + 2^52
__device__ __forceinline__ uint32_t hash_plus5_double(double a, double c, double b52) {
    const double x = __fma_rn(a, c, b52);
    const uint32_t five_hi = 5u * (uint32_t)__double2hiint(x) - 5u * MH_2_52_HI;
    uint32_t t, wrapped;
    asm("add.cc.u32 %0, %2, %3;\n\taddc.u32 %1, 0, 0;" : "=r"(t), "=r"(wrapped) : "r"((uint32_t)__double2loint(x)), "r"(five_hi));
    return t + 5u * wrapped;
}
__device__ __forceinline__ uint32_t min_plus5_short(uint32_t m, double a, double c, double b52) {
    const double x = __fma_rn(a, c, b52);
    return __viaddmin_u32(5u * (uint32_t)__double2hiint(x) + (uint32_t)__double2loint(x), 0u - 5u * MH_2_52_HI, m);
}

// Rows of MH_LIST_FROM to MH_LIST ids: two instructions and a share of others for an evaluation.  2^32 / p is a little above one, and with alpha
// the nearest whole number to a * 2^32 / p, beta that to b * 2^32 / p, y(c) = alpha * c + beta mod 2^32, one multiply-add, is the value f of the hash
// function up to an error that the id bounds:
//     y = f + e  (mod 2^32),  e = 5 * f / p + delta * c + epsilon,  |delta|, |epsilon| <= 1/2.
// A shift in beta makes e >= 0 for all ids of the row, and it stays below some e_max.  The least y of eight ids, with the number of the eight in its low bits,
// and the second of these are what a lane keeps of a row.  Of the eight of the least one, that with the least y is evaluated in full, f*: it is the row's
// minimum where every other y is at e_max or more above it, for f >= y - e_max whether y wrapped or not.  Where that does not hold (of 110 ids below
// 2^20 for a minimum in 70 to 150, in proportion to the largest id) the warp evaluates the minimum again.  Up to 32 ids that and what is set up for
// a row weigh more than is saved.  Ids from 2^MH_COL_BITS on and more than four hash functions a lane keep to the forms below, which is where the form has
// been tried out, not where it stops paying.  Those forms and this one, uniform ids, 300,000 rows of 20 to 200, 600,000 of 33, 20,000 of 1,000: 128 functions below
// 2^23 1,474 and 826 us, 967 and 765, 832 and 705, below 2^24 1,475 and 1,055, 966 and 877, 832 and 950; 160 functions below 2^16 1,002 and 772, 810
// and 948, 665 and 332, below 2^20 1,477 and 814, 1,056 and 964, 946 and 413.
// Issue and the pipes of multiply-add (two cycles) and minimum bound it.  The double forms below and this one, 128 functions: 2M Zipf sets of 20 to 200
// ids below 2^20 4,199 and 3,030 us, 300,000 below 2^16 593 and 443, below 2^22 768 and 537; 20M uniform ids below 2^20 in rows of 33 812 and
// 647, 110 705 and 344, 1,000 778 and 332.  Next to it the double forms take 8 % longer for 12 uniform ids below 2^20 a row (634 and 682),
// between 3 % less and 2 % more for other short rows.
//
// An id that a row has twice is close to itself: where rows repeat their ids nearly all minima would be evaluated again, each in more time than the double form
// takes for five functions.  A row with MH_TOO_CLOSE of them among its first 32 functions, and twice as many more as ids so many and as large lead to, is
// done in the double forms instead, and so are the warp's rows behind it.  300,000 rows of 80 ids, 128 functions, without that, with it, in the double forms
// alone: 40 ids below 2^16 twice 3,840 us, 621 and 585, below 2^20 3,849, 903 and 832, 55 and 25 of them again 2,013, 909 and 838; all different 465, 468 and 846;
// 32 functions 961, 260 and 230, all different 171, 180 and 234.
constexpr int MH_LIST = 1024;
constexpr int MH_LIST_FROM = 33;
constexpr uint32_t MH_TAG = MH_LIST / 8 - 1;
constexpr int MH_TOO_CLOSE = 6;  // of the first 32 functions
constexpr int MH_COL_BITS = 22;  // rows with ids from 2^MH_COL_BITS on take the general forms, see above
// What ids in the list are above themselves: the sum of some of them tells their number, too.
constexpr uint32_t MH_LIST_ID = 1u << 26;
struct NearParams {
    uint32_t alpha, beta;  // for ids in the list, without the shift
    uint32_t off, below;   // |delta| * p, and whether delta < 0
};
__device__ __forceinline__ NearParams near_params(uint32_t a, uint32_t b) {
    // delta = ra - 5 * a / p, and whole numbers next to it do: ra is 5 * a / 2^32 to the nearest
    const uint32_t ra = (uint32_t)((5ull * a + (1ull << 31)) >> 32), rb = (uint32_t)((5ull * b + (1ull << 31)) >> 32);
    const long long off = (long long)((uint64_t)ra * MINHASH_PRIME) - (long long)(5ull * a);  // delta * p
    return NearParams{a + ra, b + rb - (a + ra) * MH_LIST_ID, (uint32_t)llabs(off), off < 0 ? 1u : 0u};
}

// keys: [L][n_total][NW] with NW = round_key_words(4k); word j (right-aligned) = bswap32(min).
// PL = hash functions per lane per sweep; a sweep covers 32*PL consecutive hash functions and
// H > 256 takes several sweeps.  Slots past H hold a = b = 0, evaluate to 0 and are never stored,
// so the inner loop carries no predicate.
// Warps of an SM: as many as registers allow without spills that cost.  (Three and four a lane with 24 of them, in the same 80 registers: 300,000 sets of 20
// to 200 ids below 2^21 652 us and 634, of ids below 2^24 1,505 and 1,469, 400,000 of 12 ids below 2^20 284 and 276.)
template <int PL>
__global__ void __launch_bounds__(MH_THREADS, PL <= 2 ? 32 : PL <= 4 ? 22 : 18)
minhash_kernel(const int32_t* __restrict__ indices, const int32_t* __restrict__ indptr,
               const uint32_t* __restrict__ A, const uint32_t* __restrict__ B, int n_rows,
               int L, int k, int NW, uint32_t* __restrict__ keys, int n_total, int row_offset, int rows) {
    constexpr bool NEAR = PL <= 4;
    const int lane = threadIdx.x & 31;
    const int H = L * k;
    const int pad_words = NW - k;  // leading zero words when 4k is not 4, 8, 16 or 32 bytes
    __shared__ __align__(16) double ids_short[34], ids_long[34];
    __shared__ __align__(16) uint32_t ids_row[NEAR ? MH_LIST : 1];
    __shared__ __align__(16) NearParams near[NEAR ? PL : 1][32];
    bool have_near = false, repeats = false;  // the rows repeat their ids
    __shared__ size_t key_at[32 * PL];  // word of a hash function in the first row's keys
    const uint32_t below = (1u << lane) - 1u;
    double ad[PL], bd[PL];
    auto load_params = [&](int h0) {
#pragma unroll
        for (int i = 0; i < PL; ++i) {
            const int h = h0 + i * 32 + lane;
            ad[i] = h < H ? (double)A[h] : 0.0;
            bd[i] = (h < H ? (double)B[h] : 0.0) + 5.0 + MH_2_52;
            const int t = h / k;
            key_at[i * 32 + lane] = (size_t)t * n_total * NW + pad_words + (h - t * k);
        }
    };
    // The integer forms take their parameters from the doubles: these are all the loop has registers for.  Added to 2^52, as bd
    // is, an integer lies in the low bits: conversions for every 32 ids took 5 % of a row of ids from 2^20 on.
    auto a_of = [&](int i) { return (uint32_t)__double2loint(ad[i] + MH_2_52); };
    auto b5_of = [&](int i) { return (uint64_t)__double_as_longlong(bd[i]) - ((uint64_t)MH_2_52_HI << 32); };
    load_params(0);

    // the ids of a step are fetched a step ahead
    const uint32_t row0 = blockIdx.x * (uint32_t)rows;
    const int here = (int)min((uint32_t)rows, (uint32_t)n_rows - row0);
    const int bound = lane <= here ? indptr[row0 + lane] : 0;
    int start = __shfl_sync(0xFFFFFFFFu, bound, 0), end = __shfl_sync(0xFFFFFFFFu, bound, 1);
    int ahead = start + lane < end ? indices[start + lane] : 0;
    // ... and three more of a row for the near form, while the row before it is under way
    int more[3] = {0, 0, 0};
    auto fetch_more = [&](int from, int to) {
        if (NEAR && to - from >= MH_LIST_FROM && to - from <= MH_LIST) {
#pragma unroll
            for (int q = 0; q < 3; ++q) more[q] = from + 32 * (q + 1) + lane < to ? indices[from + 32 * (q + 1) + lane] : 0;
        }
    };
    fetch_more(start, end);
    for (int r = 0; r < here; ++r) {
        const int row = row_offset + (int)row0 + r;
        const int next_end = r + 1 < here ? __shfl_sync(0xFFFFFFFFu, bound, r + 2) : end;
        const uint32_t short_col = end - start <= MH_SHORT_ROW ? MH_SHORT_COL : 0u;
        bool shorts = false;  // the row has had ids below short_col
        // Rows for the near form: all ids at once, the last one again to a whole number of eights.
        const int n_ids = end - start, eights = (n_ids + 7) / 8;
        bool listed = NEAR && !repeats && n_ids >= MH_LIST_FROM && n_ids <= MH_LIST;
        uint32_t largest = 0;
        if (listed) listed = !__any_sync(0xFFFFFFFFu, (uint32_t)ahead >> MH_COL_BITS);
        if (listed) {
            largest = (uint32_t)ahead;
            ids_row[lane] = largest + MH_LIST_ID;
            auto put = [&](int at, uint32_t id) {
                if (at < n_ids) {
                    largest = max(largest, id);
                    ids_row[at] = id + MH_LIST_ID;
                }
            };
#pragma unroll
            for (int q = 0; q < 3; ++q) put(32 * (q + 1) + lane, (uint32_t)more[q]);
#pragma unroll 1
            for (int at = 128 + lane; at < n_ids; at += 32) put(at, (uint32_t)indices[start + at]);
            largest = __reduce_max_sync(0xFFFFFFFFu, largest);
            listed = largest >> MH_COL_BITS == 0;
            __syncwarp();
            if (lane < eights * 8 - n_ids) ids_row[n_ids + lane] = ids_row[n_ids - 1];
            __syncwarp();
        }
        if (r + 1 < here) fetch_more(end, next_end);
        for (int h0 = 0; h0 < H; h0 += 32 * PL) {
            const bool last = h0 + 32 * PL >= H;
            if (H > 32 * PL) load_params(h0);
            uint32_t m[PL];
#pragma unroll
            for (int i = 0; i < PL; ++i) m[i] = 0xFFFFFFFFu;
            if constexpr (NEAR) if (listed) {  // one sweep
                if (last) ahead = end + lane < next_end ? indices[end + lane] : 0;  // the next row's first
                if (!have_near) {
#pragma unroll
                    for (int i = 0; i < PL; ++i) near[i][lane] = near_params(a_of(i), (uint32_t)(b5_of(i) - 5ull));
                    have_near = true;
                }
                auto span_of = [&](const NearParams& np) { return __umulhi(np.off, largest + 1u) + 3u; };  // |delta| * largest and a little more
                uint32_t alpha[PL], beta[PL], second[PL];
#pragma unroll
                for (int i = 0; i < PL; ++i) {
                    const NearParams np = near[i][lane];
                    alpha[i] = np.alpha;
                    beta[i] = np.beta + (np.below ? span_of(np) : 1u);
                    second[i] = 0xFFFFFFFFu;
                }
                const uint4* four = reinterpret_cast<const uint4*>(ids_row);
#pragma unroll 1
                for (int j = 0; j < eights; ++j) {
                    const uint4 u = four[2 * j], v = four[2 * j + 1];
#pragma unroll
                    for (int i = 0; i < PL; ++i) {
                        auto y = [&](uint32_t c) { return alpha[i] * c + beta[i]; };
                        uint32_t t = __vimin3_u32(y(u.x), y(u.y), y(u.z));
                        t = __vimin3_u32(t, y(u.w), y(v.x));
                        t = __vimin3_u32(t, y(v.y), y(v.z));
                        t = (min(t, y(v.w)) & ~MH_TAG) | (uint32_t)j;
                        second[i] = min(second[i], max(m[i], t));
                        m[i] = min(m[i], t);
                    }
                }
                const uint32_t last_id = ids_row[n_ids - 1], times = (uint32_t)(eights * 8 - n_ids) + 1u;  // in its eight
#pragma unroll
                for (int i = 0; i < PL; ++i) {
                    const uint4 u = four[2 * (m[i] & MH_TAG)], v = four[2 * (m[i] & MH_TAG) + 1];
                    const uint32_t slack = span_of(near[i][lane]) + 8u + MH_TAG + 1u;  // e_max and what the tag takes off
                    const uint32_t base = beta[i] - (m[i] & ~MH_TAG);
                    uint32_t close = 0;  // sum of those whose y is close to the least one
                    auto look = [&](uint32_t c) { close += alpha[i] * c + base <= slack ? c : 0u; };
                    look(u.x); look(u.y); look(u.z); look(u.w);
                    look(v.x); look(v.y); look(v.z); look(v.w);
                    // The last id and its copies behind the row are one: they are all that is close where the last id is and they make up
                    // the sum.  (The sum alone does not tell: other ids around the last one have the same.)
                    if (close == last_id * times && alpha[i] * last_id + base <= slack) close = last_id;
                    const uint32_t t = hash_plus5(a_of(i), close & (MH_LIST_ID - 1u), b5_of(i));
                    // 0 where it is too close to tell, and below 5 near the prime: evaluated again
                    m[i] = close < 2u * MH_LIST_ID && t >= 5u && t <= 0xFFFFFFFFu - slack && second[i] >= t - 5u + slack ? t : 0u;
                }
                // n_ids * largest / 2^29 is what to expect
                if (__popc(__ballot_sync(0xFFFFFFFFu, m[0] == 0u && lane < H)) >= MH_TOO_CLOSE + (int)((uint32_t)n_ids * (largest >> 10) >> 18)) {
                    repeats = true;
                    listed = false;
                    ahead = indices[start + lane];
#pragma unroll
                    for (int i = 0; i < PL; ++i) m[i] = 0xFFFFFFFFu;
                }
            }
            for (int base = listed ? end : start; base < end; base += 32) {
                const int mine = ahead;
                // the next step's, then the row's first again for another sweep, or the next row's
                const bool inside = base + 32 < end;
                const int at = (inside ? base + 32 : last ? end : start) + lane;
                ahead = at < (inside || !last ? end : next_end) ? indices[at] : 0;
                const int cnt = min(32, end - base);
                if (!__any_sync(0xFFFFFFFFu, (uint32_t)mine >= MH_DOUBLE_COL)) {
                    // the two lists, the last id of an odd number twice
                    const bool have = lane < cnt, is_short = have && (uint32_t)mine < short_col;
                    const uint32_t m_short = __ballot_sync(0xFFFFFFFFu, is_short), m_long = __ballot_sync(0xFFFFFFFFu, have && !is_short);
                    const int n_short = __popc(m_short), n_long = __popc(m_long);
                    shorts = shorts || n_short > 0;
                    if (have) {
                        double* const list = is_short ? ids_short : ids_long;
                        const int at = __popc((is_short ? m_short : m_long) & below);
                        list[at] = (double)mine;
                        if (at + 1 == (is_short ? n_short : n_long)) list[at + 1] = (double)mine;
                    }
                    __syncwarp();
#pragma unroll MH_STEPS
                    for (int s = 0; s < n_short; s += 2) {
                        const double2 c = *reinterpret_cast<const double2*>(ids_short + s);
#pragma unroll
                        for (int i = 0; i < PL; ++i) m[i] = min_plus5_short(min_plus5_short(m[i], ad[i], c.x, bd[i]), ad[i], c.y, bd[i]);
                    }
                    auto two_long = [&](int s) {
                        const double2 c = *reinterpret_cast<const double2*>(ids_long + s);
#pragma unroll
                        for (int i = 0; i < PL; ++i)
                            m[i] = __vimin3_u32(m[i], hash_plus5_double(ad[i], c.x, bd[i]), hash_plus5_double(ad[i], c.y, bd[i]));
                    };
                    if (NEAR && n_long == 32) {  // rows that are too long for the list, or their ids too large, have many of these
#pragma unroll 2
                        for (int s = 0; s < 32; s += 2) two_long(s);
                    } else {
                        for (int s = 0; s < n_long; s += 2) two_long(s);
                    }
                    __syncwarp();
                    continue;
                }
                uint32_t a[PL];
                uint64_t b[PL];
#pragma unroll
                for (int i = 0; i < PL; ++i) {
                    a[i] = a_of(i);
                    b[i] = b5_of(i);
                }
                if (__any_sync(0xFFFFFFFFu, (uint32_t)mine >= MH_FAST_COL)) {
#pragma unroll (PL <= 2 ? 4 : 2)
                    for (int s = 0; s < cnt; ++s) {
                        const uint32_t c = (uint32_t)__shfl_sync(0xFFFFFFFFu, mine, s);
#pragma unroll
                        for (int i = 0; i < PL; ++i) m[i] = min(m[i], hash_plus5_any(a[i], c, b[i]));
                    }
                    continue;
                }
#pragma unroll (PL <= 4 ? 8 : 4)
                for (int s = 0; s < cnt; ++s) {
                    const uint32_t c = (uint32_t)__shfl_sync(0xFFFFFFFFu, mine, s);
#pragma unroll
                    for (int i = 0; i < PL; ++i) m[i] = min(m[i], hash_plus5(a[i], c, b[i]));
                }
            }
#pragma unroll
            for (int i = 0; i < PL; ++i) {
                uint32_t again = __ballot_sync(0xFFFFFFFFu, h0 + i * 32 + lane < H && m[i] < (shorts ? MH_AGAIN : 5u));
                while (again) {
                    const int src = __ffs(again) - 1;
                    again &= again - 1u;
                    const uint32_t a = __shfl_sync(0xFFFFFFFFu, a_of(i), src);
                    const uint32_t b = __shfl_sync(0xFFFFFFFFu, (uint32_t)(b5_of(i) - 5ull), src);
                    uint32_t exact = 0xFFFFFFFFu;
                    uint32_t plus5 = 0;
                    if constexpr (NEAR) if (listed) {  // four ids of a lane at once, the last one for those that are not there
                        plus5 = 0xFFFFFFFFu;
                        for (int e = lane; e - lane < n_ids; e += 128)
#pragma unroll
                            for (int q = 0; q < 4; ++q)
                                plus5 = min(plus5, hash_plus5(a, ids_row[min(e + 32 * q, n_ids - 1)] - MH_LIST_ID, (uint64_t)b + 5u));
                        plus5 = __reduce_min_sync(0xFFFFFFFFu, plus5);
                    }
                    if (plus5 < 5u) {
                        for (int e = start + lane; e < end; e += 32) exact = min(exact, hash_mod_prime(a, (uint32_t)indices[e], b));
                        plus5 = __reduce_min_sync(0xFFFFFFFFu, exact) + 5u;
                    }
                    if (lane == src) m[i] = plus5;
                }
                if (end > start) m[i] -= 5u;
            }
#pragma unroll
            for (int i = 0; i < PL; ++i) {
                int h = h0 + i * 32 + lane;
                if (h < H) keys[key_at[i * 32 + lane] + (size_t)row * NW] = __byte_perm(m[i], 0, 0x0123);
            }
        }
        if (end <= start) ahead = end + lane < next_end ? indices[end + lane] : 0;
        if (pad_words > 0) {
            for (int idx = lane; idx < L * pad_words; idx += 32) {
                int t = idx / pad_words, j = idx - t * pad_words;
                size_t item = (size_t)t * n_total + row;
                keys[item * NW + j] = 0u;
            }
        }
        start = end;
        end = next_end;
    }
}

inline void launch_minhash(const CtxPtr& c, cudaStream_t stream, const int32_t* indices,
                           const int32_t* indptr, const uint32_t* A, const uint32_t* B, int n_rows,
                           int L, int k, const KeySpec& ks, uint32_t* keys, int n_total,
                           int row_offset) {
    if (n_rows == 0) return;
    const int rows = (int)std::min<size_t>(MH_ROWS, ceil_div((size_t)n_rows, (size_t)c->sm_count * MH_WARPS));
    const size_t blocks = ceil_div((size_t)n_rows, (size_t)rows);
    const int H = L * k;
    const int sweeps = (int)ceil_div(H, 32 * MH_MAX_PER_LANE);
    const int per_lane = (int)ceil_div(H, 32 * sweeps);  // 1..MH_MAX_PER_LANE
#define CULSH_MH_CASE(PLV)                                                                      \
    case PLV:                                                                                   \
        minhash_kernel<PLV><<<(unsigned)blocks, MH_THREADS, 0, stream>>>(                       \
            indices, indptr, A, B, n_rows, L, k, ks.key_words, keys, n_total, row_offset, rows); \
        break;
    switch (per_lane) {
        CULSH_MH_CASE(1) CULSH_MH_CASE(2) CULSH_MH_CASE(3) CULSH_MH_CASE(4)
        CULSH_MH_CASE(5) CULSH_MH_CASE(6) CULSH_MH_CASE(7) CULSH_MH_CASE(8)
        default: fail(CULSH_ERR_INTERNAL, "minhash: hashes per lane out of range");
    }
#undef CULSH_MH_CASE
    KERNEL_CHECK();
}

}  // namespace culsh_b200
