"""Programmatic launches, checked in the sources on the CPU: a kernel that waits
for the kernel before it (pdl_wait) and every function that it calls read what
that kernel writes, so none of them has a __restrict__ parameter or uses a
read-only load (either may be moved ahead of the wait); the wait comes before any
return and any load; and every kernel that is launched programmatically waits."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "utc_gb300", "csrc")
HEAD = re.compile(r"(__global__|__device__)\b[^;{}#]*?\b(\w+)\s*\(")


def sources():
    for name in sorted(os.listdir(CSRC)):
        if name.endswith((".cu", ".cuh")):
            text = open(os.path.join(CSRC, name)).read()
            yield name, re.sub(r"//[^\n]*", "", re.sub(r"/\*.*?\*/", "", text, flags=re.S))


def close(text, at, pair):
    """Index after the bracket that closes the one at text[at]."""
    depth = 0
    for k in range(at, len(text)):
        depth += {pair[0]: 1, pair[1]: -1}.get(text[k], 0)
        if depth == 0:
            return k + 1
    raise AssertionError("unbalanced " + pair)


def functions():
    """(kind, name, file, parameters, body) of every device function and kernel."""
    out = []
    for name, text in sources():
        for m in re.finditer(r"__global__|__device__", text):
            at = m.end()
            while True:  # past __launch_bounds__(...) to the name's parameter list
                p = text.find("(", at)
                word = re.search(r"(\w+)\s*$", text[at:p])
                if word is None or word.group(1) != "__launch_bounds__":
                    break
                at = close(text, p, "()")
            if word is None:
                continue
            end = close(text, p, "()")
            tail = re.match(r"\s*(const\s*)?\{", text[end:])
            if tail is None:
                continue
            b = end + tail.end() - 1
            out.append((m.group(0), word.group(1), name, text[p:end], text[b:close(text, b, "{}")]))
    return out


def called(fns, body, seen):
    """Names of the device functions that a body calls, through any of them."""
    for kind, name, _, _, sub in fns:
        if kind == "__device__" and name not in seen and re.search(rf"\b{name}\s*(<[^;(){{}}]*>)?\s*\(", body):
            seen.add(name)
            called(fns, sub, seen)
    return seen


def test_waiting_kernels_read_through_plain_pointers():
    fns = functions()
    kernels = [f for f in fns if f[0] == "__global__" and "pdl_wait()" in f[4]]
    assert len(kernels) >= 14
    bad = set()
    for _, name, file, params, body in kernels:
        parts = [(name, file, params, body)]
        reach = called(fns, body, set())
        parts += [(n, f, p, b) for kind, n, f, p, b in fns if kind == "__device__" and n in reach]
        for n, f, p, b in parts:
            if "__restrict__" in p + b or re.search(r"__ldg|__ldlu|ld\.global\.nc", b):
                bad.add(f"{f}: {n} (of {name})")
    assert not bad, "\n".join(sorted(bad))


def test_the_wait_comes_first():
    for _, name, file, params, body in functions():
        if "pdl_wait()" not in body or name == "pdl_wait":
            continue
        before = body[:body.index("pdl_wait()")]
        assert not re.search(r"\breturn\b|__syncthreads|__shfl", before), f"{file}: {name}"
        for pointer in re.findall(r"\*\s*(\w+)", params):
            assert not re.search(rf"\b{pointer}\s*\[|\*\s*{pointer}\b", before), f"{file}: {name} reads {pointer} before the wait"


def test_programmatic_launches_are_of_waiting_kernels():
    fns = functions()
    waits = {n for kind, n, _, _, b in fns if kind == "__global__" and "pdl_wait()" in b}
    named = 0
    for name, text in sources():
        for m in re.finditer(r"pdl_launch\(\s*\"(\w+) launch\"", text):
            named += 1
            assert m.group(1) in waits, f"{name}: {m.group(1)}"
    assert named >= 14
