"""A kernel that is launched before the one in front of it is done has to wait for it before anything else, and to take all its pointers from behind
the wait; one that waits without being launched so would be harmless, but is an oversight."""
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


def _kernels(text):
    """name -> (restrict pointers, body) of every kernel."""
    out = {}
    for m in re.finditer(r"__global__ void (?:__launch_bounds__\()?", text):
        at = m.end()
        if m.group(0).endswith("("):
            at = _closing(text, at)
        name = re.compile(r"(?:\s|//[^\n]*)*(\w+)\(").match(text, at)
        end = _closing(text, name.end())
        params = re.sub(r"/\*.*?\*/", "", text[name.end():end - 1], flags=re.S)
        out[name.group(1)] = (re.findall(r"__restrict__\s+(\w+)", params), text[end:end + 4000])
    return out


def test_kernels_launched_early_wait_first():
    texts = {f: open(os.path.join(CSRC, f)).read() for f in sorted(os.listdir(CSRC))}
    kernels, early = {}, set()
    for text in texts.values():
        kernels.update(_kernels(text))
    for text in texts.values():
        for m in re.finditer(r"launch_(?:next|cluster)\((?:[\w.>-]+), (\w+)", text):
            name = m.group(1)
            if name in kernels:
                early.add(name)
                continue
            # a variable: every kernel that the function in front of the launch puts into it or could
            body = text[max(text.rfind("\ninline ", 0, m.start()), text.rfind("\nvoid ", 0, m.start()), text.rfind("\nbool ", 0, m.start())):m.start()]
            named = [k for k in re.findall(r"\b(\w+_kernel)\b(?=[<;,)\s])", body) if k in kernels]
            assigned = [k for k in re.findall(r"(?:auto\w*\s+(?:k_\w+|%s)\s*=|\bgo\(|launch_small\([^;]*?)\s*(\w+_kernel)" % name, text) if k in kernels]
            assert named or assigned, name
            early.update(k for k in assigned if k in named or not named)
    waiting = {k for k, (_, body) in kernels.items() if re.match(r"\s*\{\s*behind_kernel_before\(", body)}
    assert len(early) > 15 and early <= waiting, early - waiting
    for k in waiting:
        pointers, body = kernels[k]
        given = re.match(r"\s*\{\s*behind_kernel_before\(([^)]*)\)", body).group(1)
        assert [p for p in given.split(", ") if p][:len(pointers)] == pointers, k
    for k, (_, body) in kernels.items():  # the wait is nowhere but in front
        inside = body[:body.find("\n}\n")]
        assert inside.count("behind_kernel_before(") == (1 if k in waiting else 0), k
    # and what waits is never launched in the ordinary way
    for text in texts.values():
        for m in re.finditer(r"\b(\w+_kernel)\b(?:<[^;<>]*>)?<<<", text):
            assert m.group(1) not in waiting, m.group(1)
