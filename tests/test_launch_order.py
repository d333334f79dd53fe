"""A kernel that may be launched before the one in front of it is done takes a KernelBefore, by which the launch helpers know it.  It has to wait by it before
anything else, and to take all its pointers from behind the wait."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "culsh_b200", "csrc")


def _closing(text, at):
    """Position behind the bracket that closes the one before `at`."""
    depth = 1
    while depth:
        depth += {"(": 1, ")": -1}.get(text[at], 0)
        at += 1
    return at


def test_kernels_launched_early_wait_first():
    early = 0
    for name in sorted(os.listdir(CSRC)):
        text = re.sub(r"//[^\n]*|/\*.*?\*/", "", open(os.path.join(CSRC, name)).read(), flags=re.S)
        for m in re.finditer(r"__global__\s+void\s+(?:__launch_bounds__\s*\()?", text):
            at = _closing(text, m.end()) if m.group(0).endswith("(") else m.end()
            head = re.compile(r"\s*(\w+)\s*\(").match(text, at)
            end = _closing(text, head.end())
            params = text[head.end():end - 1]
            if "KernelBefore" not in params and "EarlyIf" not in params:
                continue
            early += 1
            assert re.search(r",\s*(?:KernelBefore|EarlyIf<\([^()]*\)>)\s+kernel_before\s*$", params), head.group(1)
            wait = re.compile(r"\s*\{\s*kernel_before\s*\.\s*wait\s*\(").match(text, end)
            assert wait, head.group(1)
            given = re.findall(r"\w+", text[wait.end():_closing(text, wait.end()) - 1])
            assert given and set(re.findall(r"__restrict__\s+(\w+)", params)) <= set(given), head.group(1)
    assert early == 25
    texts = [open(os.path.join(CSRC, name)).read() for name in sorted(os.listdir(CSRC))]  # one helper, and nothing else, asks for an early launch
    assert sum(t.count("cudaLaunchAttributeProgrammaticStreamSerialization") for t in texts) == 1
