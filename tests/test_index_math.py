"""Index arithmetic of kernels at the largest sizes the engine takes, on the CPU: no device memory of that
size is needed, or touched."""
import os
import sys

sys.path.insert(0, os.path.dirname(os.path.abspath(__file__)))
from native import run_native  # noqa: E402

TILES = r"""
#include "index_math.h"
#include <cstdio>
int main() {
    long long n, quarters, per;
    while (std::scanf("%lld %lld %lld", &n, &quarters, &per) == 3) {
        const long long total = n * quarters, tiles = (total + per - 1) / per;
        std::printf("%lld %lld %lld\n", (long long)culsh_b200::tile_first(0, (int)per),
                    (long long)culsh_b200::tile_first((uint32_t)(tiles / 2), (int)per),
                    (long long)culsh_b200::tile_first((uint32_t)(tiles - 1), (int)per));
    }
}
"""


def test_key_gather_tiles(tmp_path):
    """Keys of 4, 8 and 16 words are 1, 2 and 4 quarters of 16 bytes a row; a tile is 2,048 of them, and a table has
    fewer than 2^30 rows."""
    cases = [(n, q) for n in (1, 2048, (1 << 29) - 1, (1 << 29) + 4096, (1 << 30) - 1) for q in (1, 2, 4)]
    out = run_native(tmp_path, TILES, "".join(f"{n} {q} 2048\n" for n, q in cases)).split("\n")
    for (n, q), line in zip(cases, out):
        tiles = -(-n * q // 2048)
        assert [int(x) for x in line.split()] == [0, tiles // 2 * 2048, (tiles - 1) * 2048]


ROWS = r"""
#include "index_math.h"
#include <cstdio>
int main() {
    long long first, stride, n;
    while (std::scanf("%lld %lld %lld", &first, &stride, &n) == 3) {
        long long seen = 0, sum = 0, bad = 0;
        culsh_b200::walk_rows((uint32_t)first, (uint32_t)stride, (int)n, [&](int row) {
            ++seen;
            sum += row;
            bad += row < 0 || row >= n;
        });
        std::printf("%lld %lld %lld\n", seen, sum, bad);
    }
}
"""


def test_row_walks_end(tmp_path):
    """148 CTAs of 8 warps step by 1,184 rows: the last step of n = 2^31 - 1 rows ends beyond 2^31.  So does one of a grid that
    steps by a sixteenth of the rows."""
    top = (1 << 31) - 1
    cases = [(0, 1, 0), (0, 1184, 1), (5, 1184, 5), (7, 1184, 10_000), (1183, 1184, top), (0, 1184, top),
             (top - 1, 37_888, top), (top, 1184, top), (100, 37_888, top - 900),
             (0, -(-top // 16), top), (-(-top // 16) - 1, -(-top // 16), top), (126_250_000, 126_250_001, 2_020_000_016), (5, top, top)]
    out = run_native(tmp_path, ROWS, "".join("%d %d %d\n" % c for c in cases)).split("\n")
    for (first, stride, n), line in zip(cases, out):
        rows = range(first, n, stride)
        assert [int(x) for x in line.split()] == [len(rows), sum(rows), 0]


BLOCKS = r"""
#include "index_math.h"
#include <cstdio>
int main() {
    long long n, per;
    while (std::scanf("%lld %lld", &n, &per) == 2) std::printf("%d\n", culsh_b200::row_blocks((int)n, (int)per));
}
"""


def test_blocks_of_rows(tmp_path):
    """Blocks of 64 and 128 rows, up to n = 2^31 - 1 (queries and rows that are only hashed may be as many)."""
    top = (1 << 31) - 1
    cases = [(n, per) for per in (64, 128) for n in (1, per - 1, per, per + 1, 10 * per, top - per, top - per + 1, top - 1, top)]
    out = run_native(tmp_path, BLOCKS, "".join("%d %d\n" % c for c in cases)).split("\n")
    assert [int(x) for x in out[:len(cases)]] == [-(-n // per) for n, per in cases]
