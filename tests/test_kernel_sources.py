"""Rules of the kernels' sources that no run can show: what the compiler may assume of pointers, and index steps
that only pass 2^31 at sizes of many gigabytes."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "culsh_b200", "csrc")


def _sources():
    return {f: open(os.path.join(CSRC, f)).read() for f in sorted(os.listdir(CSRC)) if f.endswith((".cuh", ".cu", ".h"))}


def _kernels(text):
    """(name, parameters, body) of the kernels of a file."""
    for m in re.finditer(r"__global__[^;{]*?\b(\w+_kernel)\(([^)]*)\)\s*\{", text):
        depth, at = 1, m.end()
        while depth:
            depth += {"{": 1, "}": -1}.get(text[at], 0)
            at += 1
        yield m.group(1), m.group(2), text[m.end():at]


def test_host_words_are_not_read_through_a_second_pointer():
    """lookup_count_kernel makes the counters that it also leaves in host memory.  They reach it as `counters`, which
    promises that nothing else points there, and inside `host`: they are not read through the latter."""
    found = [(p, b) for t in _sources().values() for n, p, b in _kernels(t) if n == "lookup_count_kernel"]
    assert len(found) == 1
    params, body = found[0]
    assert "HostWords host" in params and re.search(r"__restrict__\s+counters\b", params)
    calls = re.findall(r"host\.write\(([^;]*)\);", body)
    assert calls and all(c.split(",")[1:] == [" s_counters"] for c in calls)


def test_blocks_of_rows_are_not_rounded_up_by_a_sum():
    """n + per - 1 passes 2^31 for the largest n: kernels count blocks of rows by row_blocks (tests/test_index_math.py)."""
    assert not [(f, n) for f, t in _sources().items() for n, _, body in _kernels(t)
                if re.search(r"\(a\.n \+ \w+ - 1\) / ", body)]


def test_rows_are_not_counted_up_in_signed_steps():
    """A step of a whole grid past the last of n < 2^31 rows may pass 2^31: rows are gone through by walk_rows, which counts unsigned
    (tests/test_index_math.py), or by an unsigned loop."""
    assert not [(f, m) for f, t in _sources().items()
                for m in re.findall(r"for \((?:int|int32_t) (?:row|q)\b[^;]*;[^;]*;[^)]*\+=[^)]*(?:gridDim|n_warps)[^)]*\)", t)]
