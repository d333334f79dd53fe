"""How the batches of a query are put together, on the CPU: every query once and in order, whole batches within the
bytes of a group, batch by batch after a group that has too many entries or finds no memory, and
errors of a single batch passed on."""
import os
import sys

import pytest

sys.path.insert(0, os.path.dirname(os.path.abspath(__file__)))
from native import run_native  # noqa: E402

CUDA = "/usr/local/cuda/include"
pytestmark = pytest.mark.skipif(not os.path.exists(os.path.join(CUDA, "cuda_runtime_api.h")), reason="no CUDA headers")

PROGRAM = r"""
#include "query_groups.h"
#include <cstdio>
using namespace culsh_b200;
extern "C" const char* cudaGetErrorString(cudaError_t) { return ""; }
// fail: 0 nothing, 1 too many entries, 2 no memory, 3 another error, 4 no memory in every call; at: in calls from this query on
int main() {
    int n_q, batch, L, words, fail_how, at;
    while (std::scanf("%d %d %d %d %d %d", &n_q, &batch, &L, &words, &fail_how, &at) == 6) {
        const int group = query_group(n_q, batch, L, words);
        std::printf("%d", group);
        int released = 0;
        try {
            run_query_groups(n_q, batch, group, GROUP_IDS, [&](int s0, int nb, uint64_t limit) {
                const bool hit = s0 + nb > at && (nb > batch || fail_how >= 3);
                if ((nb > batch) != (limit == GROUP_IDS)) fail(CULSH_ERR_INTERNAL, "limit");
                if (hit && fail_how == 1) return false;
                if (hit && (fail_how == 2 || fail_how == 4)) fail(CULSH_ERR_ALLOC, "none left");
                if (hit && fail_how == 3) fail(CULSH_ERR_CUDA, "broken");
                std::printf(" %d:%d", s0, nb);
                return true;
            }, [&] { ++released; });
        } catch (const Error& e) {
            std::printf(" error %d", e.status);
        }
        std::printf(" released %d\n", released);
    }
}
"""


def _run(tmp_path, cases):
    out = run_native(tmp_path, PROGRAM, "".join("%d %d %d %d %d %d\n" % c for c in cases), flags=["-I", CUDA])
    return out.strip().split("\n")


def _parts(line):
    return [tuple(int(x) for x in p.split(":")) for p in line.split()[1:] if ":" in p]


@pytest.mark.parametrize("words", [1, 2, 4, 8, 16])
def test_groups_hold_whole_batches_within_their_bytes(tmp_path, words):
    cases = [(n, b, L, words, 0, 0) for L in (1, 24, 100_000, 30_000_000) for n, b in
             ((1, 1), (10, 3), (100_003, 10_000), (1 << 21, 64), ((1 << 31) - 1, 1 << 30), ((1 << 31) - 1, (1 << 31) - 2))]
    for (n, b, L, w, _, _), line in zip(cases, _run(tmp_path, cases)):
        group = int(line.split()[0])
        assert group == n or group % b == 0
        assert group <= b or group * L * (4 * w + 9) <= 52 << 20
        at = 0
        for s0, nb in _parts(line):
            assert s0 == at and nb == min(group, n - at)
            at += nb
        assert at == n and line.endswith("released 0")


def test_what_a_group_cannot_do_goes_batch_by_batch(tmp_path):
    n, b = 1003, 100
    whole, entries, memory, late, other, every = _run(tmp_path, [
        (n, b, 24, 1, 0, 0), (n, b, 24, 1, 1, 0), (n, b, 24, 1, 2, 0), (1 << 20, b, 24, 1, 2, 500_000), (n, b, 24, 1, 3, 0), (n, b, 24, 1, 4, 0)])
    single = [(s, min(b, n - s)) for s in range(0, n, b)]
    assert _parts(whole) == [(0, n)] and whole.endswith("released 0")
    assert _parts(entries) == single and entries.endswith("released 0")
    assert _parts(memory) == single and memory.endswith("released 1")
    parts = _parts(late)
    assert parts[0][1] > b and all(nb <= b for _, nb in parts[parts.index(next(p for p in parts if p[1] == b)):])
    assert sum(nb for _, nb in parts) == 1 << 20 and late.endswith("released 1")
    assert "error" in other and not _parts(other) and other.endswith("released 0")
    assert "error" in every and not _parts(every) and every.endswith("released 1")


WIDE = r"""
#include "query_groups.h"
#include <cstdio>
using namespace culsh_b200;
extern "C" const char* cudaGetErrorString(cudaError_t) { return ""; }
int main() {
    int n_q, L, memory;
    while (std::scanf("%d %d %d", &n_q, &L, &memory) == 3) {
        std::printf("%d", query_is_wide(n_q, L) ? 1 : 0);
        try {
            run_query_groups(n_q, n_q - n_q / 2, n_q, UINT64_MAX, [&](int s0, int nb, uint64_t limit) {
                if (limit != UINT64_MAX) fail(CULSH_ERR_INTERNAL, "limit");
                if (nb > memory) fail(CULSH_ERR_ALLOC, "none left");
                std::printf(" %d:%d", s0, nb);
                return true;
            }, [] {});
        } catch (const Error& e) {
            std::printf(" error %d", e.status);
        }
        std::printf("\n");
    }
}
"""


def test_a_wide_query_goes_in_halves_when_memory_is_short(tmp_path):
    top = (1 << 31) - 1
    cases = [(1 << 20, 1024, top), ((1 << 20) + 1, 1024, top), ((1 << 20) + 1, 1024, 1 << 20), (top, 1, 1 << 30), (top, 1, 5)]
    out = run_native(tmp_path, WIDE, "".join("%d %d %d\n" % c for c in cases), flags=["-I", CUDA]).strip().split("\n")
    assert [int(line.split()[0]) for line in out] == [0, 1, 1, 1, 1]
    half = ((1 << 20) + 2) // 2
    assert _parts(out[1]) == [(0, (1 << 20) + 1)]
    assert _parts(out[2]) == [(0, half), (half, half - 1)]
    assert _parts(out[3]) == [(0, 1 << 30), (1 << 30, (1 << 30) - 1)]
    assert "error" in out[4] and not _parts(out[4])
