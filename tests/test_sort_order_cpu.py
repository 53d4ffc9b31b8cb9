"""The step of the sort that no run has been seen to need: ranks that came out of lane order are found and put right.
Its code, compiled for the host, against a stable sort."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from conftest import ROOT


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("sortorder") / "libsort_order_host.so")
    subprocess.check_call(["g++", "-std=c++17", "-O2", "-shared", "-fPIC", "-o", so,
                           os.path.join(ROOT, "tests", "hostmath", "sort_order_host.cpp")])
    lib = ctypes.CDLL(so)
    lib.host_out_of_order.argtypes = [ctypes.c_void_p, ctypes.c_int, ctypes.c_int, ctypes.c_uint32]
    lib.host_put_right.argtypes = lib.host_out_of_order.argtypes + [ctypes.c_int, ctypes.c_int]
    return lib


def _tile(rng, count, digits, shift, bits):
    """Packed words of a tile, in the order in which its warps hold them: the digits done and the index below
    ``shift`` ascend (the passes before have seen to that), the digit and what is above it are random."""
    below = np.sort(rng.choice(1 << min(shift, 40), size=count, replace=False).astype(np.uint64))
    digit = rng.integers(0, digits, size=count).astype(np.uint64) if digits else np.zeros(count, np.uint64)
    above = rng.integers(0, 1 << max(0, min(62 - shift - bits, 20)), size=count).astype(np.uint64)
    return (above << np.uint64(shift + bits)) | (digit << np.uint64(shift)) | below, digit


def _served(rng, words, digit, kind):
    """The tile ordered by digit with ranks in the order in which the lanes of each instruction (32 elements) were
    served: as they stand, backwards, or at random."""
    lane_order = {"straight": lambda m: np.arange(m), "backwards": lambda m: np.arange(m)[::-1],
                  "random": lambda m: rng.permutation(m), "one pair": None}[kind]
    at = np.arange(len(words))
    if kind == "one pair":
        for g in range(0, len(words) - 32, 1024):
            pair = np.flatnonzero(digit[g:g + 32] == digit[g]) + g
            if len(pair) > 1:
                at[pair[:2]] = at[pair[1::-1]]
    else:
        for g in range(0, len(words), 32):
            m = min(32, len(words) - g)
            at[g:g + m] = g + lane_order(m)
    order = at[np.argsort(digit[at], kind="stable")]
    return np.ascontiguousarray(words[order])


@pytest.mark.parametrize("count", [1, 2, 31, 33, 4095, 4096, 8191, 8192])
@pytest.mark.parametrize("digits", [1, 2, 7, 1024])
@pytest.mark.parametrize("kind", ["straight", "one pair", "backwards", "random"])
def test_ranks_out_of_lane_order_are_put_right(lib, count, digits, kind):
    rng = np.random.default_rng(count * 8 + digits)
    for shift, bits in ((23, 10), (14, 9), (53, 10)):       # first digit, a middle one of few points, the topmost
        digits_here, mask = min(digits, 1 << bits), (1 << bits) - 1
        words, digit = _tile(rng, count, digits_here, shift, bits)
        want = words[np.argsort(digit, kind="stable")]
        got = _served(rng, words, digit, kind)
        assert bool(lib.host_out_of_order(got.ctypes.data, count, shift, mask)) == (not np.array_equal(got, want))
        for backwards in (0, 1):
            tile = got.copy()
            rounds = lib.host_put_right(tile.ctypes.data, count, shift, mask, 512, backwards)
            assert 0 <= rounds <= 17                        # 32 lanes: 32 phases, and the round that finds nothing
            assert np.array_equal(tile, want)


@pytest.mark.parametrize("count", [2, 3, 513, 8192])
def test_the_rounds_suffice_for_any_disorder(lib, count):
    rng = np.random.default_rng(count)
    words, digit = _tile(rng, count, 1, 23, 10)
    tile = np.ascontiguousarray(words[::-1])
    assert lib.host_put_right(tile.ctypes.data, count, 23, 1023, 512, 0) >= 0
    assert np.array_equal(tile, words)
