"""Rules that the CUDA sources keep and that no run shows to be broken: checked on the text."""
import glob
import os
import re

import pytest

from conftest import ROOT

SOURCES = sorted(glob.glob(os.path.join(ROOT, "pointtransformerv3_b200", "csrc", "*.cu*")))


def _code(path):
    text = open(path).read()
    return re.sub(r"//[^\n]*", "", re.sub(r"/\*.*?\*/", "", text, flags=re.S))


def _to_matching(text, start, pair):
    """End of the bracketed text that opens at or after ``start``."""
    i = text.index(pair[0], start)
    depth = 0
    while True:
        depth += {pair[0]: 1, pair[1]: -1}.get(text[i], 0)
        i += 1
        if depth == 0:
            return i


def _kernels(text):
    """(name, parameters, body) of every kernel that the text defines."""
    for m in re.finditer(r"__global__\s+void\s+", text):
        at = m.end()
        if text.startswith("__launch_bounds__", at):
            at = _to_matching(text, at, "()")
        name = re.match(r"\s*(\w+)", text[at:]).group(1)
        end = _to_matching(text, text.index(name, at), "()")
        if text[end:].lstrip().startswith("{"):
            yield name, text[at:end], text[end:_to_matching(text, end, "{}")]


@pytest.mark.parametrize("path", SOURCES, ids=os.path.basename)
def test_kernels_that_start_early_read_through_plain_pointers(path):
    """A kernel that waits for the one ahead of it (pdl_wait) must not load ahead of that wait what the other
    writes.  A memory clobber holds back loads through plain pointers only: one through const __restrict__, or
    __ldg, says that nothing writes there while the kernel runs, and may be moved ahead of it."""
    text = _code(path)
    waiting = [k for k in _kernels(text) if "pdl_wait()" in k[2]]
    assert len(waiting) > 0 or "pdl_wait()" not in text or os.path.basename(path) == "common.cuh"
    for name, parameters, body in waiting:
        for word in ("__restrict__", "__ldg", "ld.global.nc"):
            assert word not in parameters + body, "%s in %s" % (word, name)
    if waiting:          # nor do the functions they are made of
        for m in re.finditer(r"__device__ __forceinline__[^{;]*", text):
            assert "__restrict__" not in m.group(0), m.group(0)
