"""What orders the kernels' accesses, checked in the sources: a race shows in few runs, so the rule is
tested where it stands instead of its rare result."""
import os
import re

from rustyfem_b200 import _build


def source(name):
    with open(os.path.join(_build.CSRC, name)) as f:
        return re.sub(r"//[^\n]*", "", f.read())


def body(text, kernel):
    """The kernel's body, braces matched."""
    i = text.index("{", re.search(r"\b" + kernel + r"\s*\(", text).end())
    depth = 0
    for j in range(i, len(text)):
        depth += {"{": 1, "}": -1}.get(text[j], 0)
        if depth == 0:
            return text[i:j + 1]
    raise ValueError(kernel)


def test_pivot_block_is_read_before_it_is_replaced():
    # every lane of warps 0 and 1 loads the sub-panel's 8×8 diagonal block, one thread of warp 1 stores
    # its factor in its place: a barrier of both warps stands between
    b = body(source("numeric.cu"), "k_pivot_block")
    load = max(m.end() for m in re.finditer(r"reinterpret_cast<const double2\*>\(A \+ \(c0 \+ i\)", b))
    store = b.index("if (tid == 32)")
    bar = b.index('bar.sync 1, 64;')
    assert load < bar < store
    assert b.rindex("if (warp < 2)", 0, bar) > b.rindex("__syncthreads()", 0, bar)
