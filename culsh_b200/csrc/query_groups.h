// Batches of a query.  A batch bounds the temporaries of a call.  Batches that are far below what is worth
// bounding share their launches and waits: as many whole ones as GROUP_BYTES of query keys and lists hold,
// unless their lists turn out to have more than GROUP_IDS entries, or memory is short; then each goes
// by itself.  100,003 queries in batches of 10,000 (24 tables, 1.7 M ids a batch): 1.94 -> 0.56 ms.
#pragma once

#include <algorithm>
#include <cstdint>

#include "check.h"

namespace culsh_b200 {

constexpr int64_t GROUP_BYTES = (int64_t)52 << 20;  // 4 M lists with keys of one word, 0.7 M with sixteen
constexpr uint64_t GROUP_IDS = (uint64_t)32 << 20;  // 128 MB

// Queries that are taken at once: whole batches, one at least.
inline int query_group(int n_q, int batch, int L, int key_words) {
    const int64_t lists = GROUP_BYTES / (4 * key_words + 9);  // key, list and range flag of a (table, query) pair
    return (int)std::min<int64_t>(n_q, std::max<int64_t>(1, lists / L / batch) * batch);
}

// A query of more (table, query) pairs than this that asks for no batches holds 8 bytes a pair for its lists, 8.6 to
// 17 GB; when there is no memory for that it goes in two halves.
inline bool query_is_wide(int n_q, int L) { return (uint64_t)n_q * (uint64_t)L > ((uint64_t)1 << 30); }

// Calls run(first query, queries, most list entries) until n_q are done, `group` at a time; when that is more than
// a batch and run gives it up (false; most entries: `group_ids`) or finds no memory (CULSH_ERR_ALLOC, after which
// release() is called), these and all that follow go batch by batch.
template <typename Run, typename Release>
inline void run_query_groups(int n_q, int batch, int group, uint64_t group_ids, Run&& run, Release&& release) {
    for (int64_t s0 = 0; s0 < n_q;) {
        const int nb = (int)std::min<int64_t>(group, n_q - s0);
        bool done = false;
        try {
            done = run((int)s0, nb, nb > batch ? group_ids : UINT64_MAX);
        } catch (const Error& e) {
            if (e.status != CULSH_ERR_ALLOC || nb <= batch) throw;
            release();
        }
        if (done) s0 += nb;
        else group = batch;
    }
}

}  // namespace culsh_b200
