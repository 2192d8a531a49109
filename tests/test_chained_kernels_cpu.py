"""Rules of the kernels that may start under the tail of the one before them (launch_chained), read off their sources."""
import os
import re

import pytest

from rapid_h3_b200 import _build


def kernels(name):
    """{kernel name: (parameter list, body)} of every __global__ function of csrc/<name>, comments left out."""
    text = open(os.path.join(_build.CSRC, name)).read()
    text = re.sub(r"//[^\n]*", "", text)
    out = {}
    for m in re.finditer(r"__global__[^;{]*?\b(\w+_kernel)\s*\(", text):
        at, depth = m.end(), 1
        while depth:
            depth += {"(": 1, ")": -1}.get(text[at], 0)
            at += 1
        params, start = text[m.end():at - 1], text.index("{", at)
        at, depth = start + 1, 1
        while depth:
            depth += {"{": 1, "}": -1}.get(text[at], 0)
            at += 1
        out[m.group(1)] = (params, text[start:at])
    return out


CHAINED = [(f, k) for f in _build.sources() for k, (_, body) in kernels(f).items() if "grid_dependency_" in body]


def test_the_chained_kernels_are_found():
    launched = sum(len(re.findall(r"launch_(?:chained|kernel)\(", open(os.path.join(_build.CSRC, f)).read())) for f in _build.sources())
    assert len(CHAINED) >= 15 and launched >= len(CHAINED)


@pytest.mark.parametrize("source,kernel", CHAINED)
def test_tensor_memory_is_allocated_before_the_next_kernel_may_start(source, kernel):
    """A kernel that lets the next one start and allocates afterwards could find the tensor memory of its SM taken by a kernel
    that waits for it in its turn."""
    body = kernels(source)[kernel][1]
    if "tmem_alloc" in body:
        triggers = [m.start() for m in re.finditer(r"grid_dependency_(begin|trigger)\(", body)]
        assert triggers and body.index("tmem_alloc") < min(triggers)


# what a chained kernel may read as read-only data: norm weights and affine parameters, rope tables
CONSTANTS = r"(?:w|p\.w|p\.act_w|gamma|beta|tab|tab_words)"


@pytest.mark.parametrize("source", sorted({f for f, _ in CHAINED}))
def test_what_the_kernel_before_wrote_is_read_by_ordinary_loads(source):
    """__ldg and `const __restrict__` promise that the data stay as they are for the kernel's lifetime, which begins while the
    kernel before it may still write them: chained kernels make that promise for constants only."""
    text = re.sub(r"//[^\n]*", "", open(os.path.join(_build.CSRC, source)).read())
    for kernel, (params, body) in kernels(source).items():
        if (source, kernel) in CHAINED:
            promised = re.findall(r"const\s+\w+\s*\*\s*__restrict__\s+(\w+)", params)
            assert all(re.fullmatch(CONSTANTS, n) for n in promised), (kernel, promised)
        else:
            text = text.replace(body, "")
    for arg in re.findall(r"__ldg\((.*)", text):
        name = re.match(r"(?:reinterpret_cast<[^>]*>\()?([\w.]+)", arg).group(1)
        assert re.fullmatch(CONSTANTS, name), arg
