"""Loads of the kernels that may start before the launch that writes their
vector has finished, checked in the sources.

Such a kernel may read the gathered x, t and G2 only with loads that stay
coherent and behind griddepcontrol.wait: ordinary ones, or bulk copies after a
proxy fence.  __ldg and const __restrict__ parameters are for data that no
launch writes (block data, descriptors, runs, permutations).  Wrong loads may
well give right results (they did), so this is a check of the text.
"""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "bigwham_dev_b200", "csrc")


def _body(file, function):
    """Parameters and body of a function, comments taken out."""
    with open(os.path.join(CSRC, file)) as f:
        src = re.sub(r"//[^\n]*", "", f.read())
    at = src.index(function + "(")
    brace = src.index("{", src.index(")", at))
    depth, end = 0, brace
    while True:
        depth += {"{": 1, "}": -1}.get(src[end], 0)
        end += 1
        if depth == 0:
            return src[at:brace], src[brace:end]


@pytest.mark.parametrize("file,function,read", [
    ("bw_kernels.cuh", "void narrow_fma_chunk", r"g\[cq\]"),
    ("bw_kernels.cuh", "void narrow_bf16_chunk_t", r"unpack_hilo\(g\[c\]\)"),
    ("bw_kernels.cuh", "void gather_g2_kernel", r"\(\(rf >> 31\) \? t : xp\)\[ro \+ k\]"),
    ("bw_multi_kernels.cuh", "narrow_multi_kernel", r"\bxr\[p\]")])
def test_vectors_are_read_with_coherent_loads(file, function, read):
    params, body = _body(file, function)
    assert len(re.findall(read, body)) == 1
    assert not re.search(r"__ldg\((g|xr|xk|tk|xp|t|a\.gsrc)\b", body)
    for name in ("xp", "t", "g2", "g"):
        assert not re.search(r"__restrict__\s+" + name + r"\b", params)


@pytest.mark.parametrize("file,function", [("bw_kernels.cuh", "stream_panels_kernel"),
                                           ("bw_multi_kernels.cuh", "stream_multi_kernel"),
                                           ("bw_mm_kernels.cuh", "mm_stream_kernel")])
def test_bulk_copies_come_after_a_proxy_fence(file, function):
    _, body = _body(file, function)
    fence = r"pdl_wait\(\);\s*fence_proxy_async_global\(\);\s*pdl_launch_dependents\(\);"
    assert len(re.findall(fence, body)) == 1
    assert len(re.findall(r"fence_proxy_async_global|pdl_launch_dependents", body)) == 2
