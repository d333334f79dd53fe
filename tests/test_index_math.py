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
