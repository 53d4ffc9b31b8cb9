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
    """(first character, end, body) of every kernel that the text defines."""
    for m in re.finditer(r"__global__\s+void\s+", text):
        at = m.end()
        if text.startswith("__launch_bounds__", at):
            at = _to_matching(text, at, "()")
        end = _to_matching(text, at, "()")
        if text[end:].lstrip().startswith("{"):
            stop = _to_matching(text, end, "{}")
            yield m.start(), stop, text[end:stop]


WORDS = ("__restrict__", "__ldg", "ld.global.nc")


def _functions_with_such_loads():
    """Names of the functions in headers that declare their loads free of writers."""
    names = set()
    for path in SOURCES:
        if path.endswith(".cuh"):
            text = _code(path)
            for first, end, _ in reversed(list(_kernels(text))):
                text = text[:first] + text[end:]
            for m in re.finditer(r"__device__[^;{}()]*?(\w+)\(", text):
                end = _to_matching(text, _to_matching(text, m.end() - 1, "()"), "{}")
                if any(w in text[m.start():end] for w in WORDS):
                    names.add(m.group(1))
    return names


@pytest.mark.parametrize("path", [p for p in SOURCES if p.endswith(".cu")], ids=os.path.basename)
def test_kernels_that_start_early_read_through_plain_pointers(path):
    """A kernel that waits for the one ahead of it (pdl_wait) must not load ahead of that wait what the other
    writes.  A memory clobber holds back loads through plain pointers only: one through const __restrict__, or
    __ldg, says that nothing writes there while the kernel runs, and may be moved ahead of it.  The same holds for the
    functions that such kernels call."""
    text = _code(path)
    kernels = list(_kernels(text))
    waits = [body for _, _, body in kernels if "pdl_wait()" in body]
    assert waits or "pdl_wait()" not in text
    for name in _functions_with_such_loads():
        assert not any(re.search(r"\b%s\(" % name, body) for body in waits), name
    if waits:
        for first, end, body in reversed(kernels):
            if "pdl_wait()" not in body:                 # an ordinary launch: free to say so
                text = text[:first] + text[end:]
        for word in WORDS:
            at = text.find(word)
            assert at < 0, text[max(0, at - 200):at + 100]
