// Which tensor-core kernel projects a shape, and in which chunks of hash columns.  Host code only.
#pragma once

#include <algorithm>
#include <cstddef>
#include <cstdlib>

namespace culsh_b200 {

// accumulator columns of a chunk at most: operands in shared memory (max MMA N), rows in tensor
// memory, and the wide form of the latter (shapes of several chunks)
constexpr int TC_BN = 256;
constexpr int TS_BN = 128;
constexpr int TS_BN_WIDE = 192;

struct TcPlan {
    int kblk, d_pad, n_chunks, tables_per_chunk, n_mma, bn;
    bool ts;
};

inline int tc_kblk_choice() {
    static int v = [] {
        const char* e = getenv("CULSH_TC_KBLK");
        int k = e ? atoi(e) : 16;
        return k == 32 ? 32 : 16;
    }();
    return v;
}

// Which kernel projects a shape.  Three forms: both operands in shared memory with chunks of
// <= 256 hash columns (project_tc_kernel), X in tensor memory with chunks of <= 128 columns, or of
// <= 192 columns (project_ts_kernel).  Measured on B200 (fit, ms):
//                                        shared, 256   tensor, 128   tensor, 192
//   12.5M x 96,  16 x 8  (one chunk)         2.31          1.85           -
//   1M x 128,    32 x 16                     0.62          0.66          0.62
//   10M x 256,   48 x 24                     24.8          29            22.7
// One chunk: the 128-column form.  Several chunks: see tc_tensor_is_cheaper.
// CULSH_TC_VARIANT (read once per process) overrides: 0 = shared memory always, 1 = tensor memory /
// 128 columns wherever it applies, 3 = tensor memory / 192 columns for shapes of several chunks
// (the tests run every shape through each).
inline int tc_variant() {
    static int v = [] {
        const char* e = getenv("CULSH_TC_VARIANT");
        return e && *e ? atoi(e) : 2;
    }();
    return v;
}

inline void tc_chunking(int L, int k, int bn, int& tables_per_chunk, int& n_chunks, int& n_mma) {
    tables_per_chunk = std::min(L, bn / k);
    n_chunks = (L + tables_per_chunk - 1) / tables_per_chunk;
    // Evenly: a chunk of few tables costs as much as a full one.  22 x 13 hashes are two chunks of 144
    // columns instead of 256 and 39 padded to 256; 24 x 18 two of 224 (100,003 x 96 rows: 56.4 -> 55.2 us).
    tables_per_chunk = (L + n_chunks - 1) / n_chunks;
    n_mma = (tables_per_chunk * k + 15) / 16 * 16;
}

// Several chunks: tensor memory with chunks of <= 192 columns, or shared memory with <= 256.  A unit
// (128 rows x a chunk) takes as long as its MMAs or, with few features, as its epilogue; nanoseconds fitted
// to 34 shapes of 160 to 1,536 columns at 32 to 1,024 features, each in both forms (RPLSH, 60,000 to
// 500,000 rows).  Over these the cheaper form by this estimate is at most 1.8 % slower than the faster one;
// estimating MMAs alone, with one factor for the epilogue's share, took 41 x 30 hashes at 256 features
// into shared memory, 737 us against 664.
inline bool tc_tensor_is_cheaper(int d, int L, int k) {
    auto cost = [&](int bn, double per_feature, double per_feature_column) {
        int tables, chunks, columns;
        tc_chunking(L, k, bn, tables, chunks, columns);
        return chunks * std::max(d * (per_feature + per_feature_column * columns), 750.0 + 6.8 * columns);
    };
    return cost(TS_BN_WIDE, 17.4, 0.040) < 1.02 * cost(TC_BN, 22.2, 0.047);
}

inline bool tc_plan(int d, int L, int k, TcPlan& p) {
    const int variant = tc_variant();
    bool ts;
    int bn;
    if (variant == 0) { ts = false; bn = TC_BN; }
    else if (variant == 1) { ts = k <= TS_BN; bn = ts ? TS_BN : TC_BN; }
    else if (variant == 3) { ts = k <= TS_BN_WIDE; bn = ts ? (L * k > TS_BN ? TS_BN_WIDE : TS_BN) : TC_BN; }
    else if (L * k <= TS_BN) { ts = true; bn = TS_BN; }
    else {
        ts = k <= TS_BN_WIDE && tc_tensor_is_cheaper(d, L, k);
        bn = ts ? TS_BN_WIDE : TC_BN;
    }
    p.bn = bn;
    if (k > bn || d % 4 != 0) return false;
    p.ts = ts;
    p.kblk = ts ? 32 : tc_kblk_choice();
    p.d_pad = (d + p.kblk - 1) / p.kblk * p.kblk;
    tc_chunking(L, k, bn, p.tables_per_chunk, p.n_chunks, p.n_mma);
    return true;
}

// hi and lo part of the projection in the layout of the plan
inline size_t tc_split_bytes(const TcPlan& p) { return sizeof(float) * (size_t)p.n_chunks * 2 * p.n_mma * p.d_pad; }

}  // namespace culsh_b200
