"""What orders the kernels' accesses, checked in the sources: a race shows in few runs, so the rule is
tested where it stands instead of its rare result."""
import os
import re

import pytest

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


# constant while a chain of programmatic launches runs: the plan's arrays, the source values, the TMA
# descriptors
PLAN = {"fr", "order", "pre", "pre_tiles", "pre_a", "pre_scr", "pre_scr_prev", "pre_panel", "pre_part", "rows",
        "imap", "mode", "omode", "slots", "items", "colbase", "chain_blk", "dst", "seg_ptr", "seg_src", "src",
        "width", "cmaps"}
# and during the sweeps the factor
FACTOR = {"panel", "linv", "inv", "d"}


def chained_kernels(name):
    """(kernel, parameter list, body) of the kernels that wait for a programmatic predecessor."""
    text = source(name)
    for m in re.finditer(r"__global__.*?\b(k_\w+)\s*\(", text, re.S):
        i, depth = m.end(), 1
        while depth:
            depth += {"(": 1, ")": -1}.get(text[i], 0)
            i += 1
        b = body(text[m.start():], m.group(1))
        if "pdl_wait()" in b:
            yield m.group(1), text[m.end():i - 1], b


@pytest.mark.parametrize("name,constant", [("numeric.cu", PLAN), ("kernels_tc.cu", PLAN),
                                           ("solve.cu", PLAN | FACTOR), ("chain.cu", PLAN | FACTOR)])
def test_chained_kernels_read_coherently(name, constant):
    # a kernel launched early lives beside the kernels that write its inputs: const __restrict__ (which lets
    # the compiler take the non-coherent path) and __ldg only for what is constant for the whole chain
    kernels = list(chained_kernels(name))
    assert kernels
    for k, params, b in kernels:
        found = set(re.findall(r"const\s+\w+\s*\*\s*__restrict__\s+(\w+)", params))
        assert found <= constant, (k, found - constant)
        assert set(re.findall(r"__ldg\((\w+)", b)) <= constant, k
