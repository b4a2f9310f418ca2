"""CPU-side checks, on the sources, of the rules a kernel keeps that may start while the kernel before it still runs."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "sptorch_b200", "csrc")


def _source(name):
    text = open(os.path.join(CSRC, name)).read()
    return re.sub(r"//[^\n]*", "", re.sub(r"/\*.*?\*/", "", text, flags=re.S))


def _block(text, at):
    """The braces' contents that open at text[at]."""
    depth = 0
    for i in range(at, len(text)):
        depth += {"{": 1, "}": -1}.get(text[i], 0)
        if depth == 0:
            return text[at + 1:i]
    raise AssertionError("unbalanced braces")


def _kernels(name):
    """[(kernel, parameter list, body)] of the file's kernels that wait for their predecessor themselves."""
    text, out = _source(name), []
    for m in re.finditer(r"__global__[^;{]*?(\w+_kernel)\s*\(([^{]*?)\)\s*\{", text):
        body = _block(text, m.end() - 1)
        if "pdl_acquire()" in body:
            out.append((m.group(1), m.group(2), body))
    return out


def test_row_operations_read_nothing_ahead_of_the_wait():
    """These kernels serve the public operations as well as the models: any operand, norm weights included, may be what the kernel before
    has just written."""
    kernels = _kernels("rowops.cu") + _kernels("rope.cu")
    assert len(kernels) >= 6
    for kernel, params, body in kernels:
        pointers = re.findall(r"\*\s*(?:__restrict__\s+)?(\w+)", params)
        ahead = body[:body.index("pdl_acquire()")]
        for p in set(pointers) - {"status"}:
            assert not re.search(r"(?<![.\w])%s\b" % p, ahead), f"{kernel} reads {p} ahead of its wait"
