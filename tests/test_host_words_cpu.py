"""Mapped host words that a kernel reports a result in: who may clear them, and when."""
import ctypes

from pointtransformerv3_b200 import ops


class Kernels:
    """Stands in for the library: "kernels" launched on a stream store their result when the host waits for it
    (in launch order, as a stream runs them)."""

    def __init__(self, words):
        self.words, self.queued = words, []

    def launch(self, value):
        self.queued.append(value)

    def ptv3_host_wait(self, last, stream):
        assert last == ctypes.addressof(self.words) + 8 * (len(self.words) - 1)
        while not self.words[len(self.words) - 1]:
            self.words[0] = self.queued.pop(0)
            self.words[len(self.words) - 1] = 1
        return 0


def host_words(n):
    host = ops._HostWords.__new__(ops._HostWords)
    host.words = (ctypes.c_int64 * n)()
    host.last = ctypes.addressof(host.words) + 8 * (n - 1)
    return host, Kernels(host.words)


def test_result_given_up_is_not_taken_for_the_next_one():
    host, lib = host_words(3)
    for value, given_up in ((5, False), (6, True), (7, True), (8, False), (9, False)):
        host.begin(lib, 0)
        assert not any(v in (6, 7) for v in lib.queued), "a kernel that nobody waited for still owns the words"
        lib.launch(value)
        host.launched(0, "kernel")
        if not given_up:
            assert host.wait(lib, 0)[0] == value and not host.pending
    assert not lib.queued


def test_launch_that_failed_is_not_waited_for():
    host, lib = host_words(2)
    host.begin(lib, 0)                   # the launch raises: no kernel will ever store anything
    host.begin(lib, 0)
    lib.launch(3)
    host.launched(0, "kernel")
    assert host.wait(lib, 0)[0] == 3
