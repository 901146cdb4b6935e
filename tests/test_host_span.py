"""The rule by which a kernel may copy to and from a caller's host buffer itself
(fluidsim_gb300/csrc/fsim_span.h), compiled for the CPU.

A buffer may begin in one page-locked allocation and end in another with pages in
between that the device cannot reach, so both ends being page-locked is not
enough.  Such a buffer is never handed to the GPU here.
"""
import ctypes as C
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "fluidsim_gb300", "csrc")
WRAPPER = """
#include "fsim_span.h"
extern "C" int addressable(int host, uintptr_t dev, uintptr_t start, size_t size, size_t bytes)
{
    return fsim_rt::span_addressable({host != 0, dev, start, size}, bytes);
}
"""
PAGE = 4096


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("span")
    src, so = str(d / "span.cpp"), str(d / "span.so")
    with open(src, "w") as f:
        f.write(WRAPPER)
    subprocess.check_call(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-I", CSRC, src, "-o", so])
    f = C.CDLL(so).addressable
    f.argtypes = [C.c_int, C.c_size_t, C.c_size_t, C.c_size_t, C.c_size_t]
    return f


def _query(ranges, p):
    """What the driver answers for address p with these page-locked (start, size) ranges."""
    for start, size in ranges:
        if start <= p < start + size:
            return 1, p, start, size
    return 0, 0, 0, 0


def test_buffers_against_every_byte(lib):
    ranges = [(16 * PAGE, 2 * PAGE), (20 * PAGE, PAGE), (21 * PAGE, 3 * PAGE)]  # a hole, then two that touch
    locked = lambda p: any(s <= p < s + n for s, n in ranges)  # noqa: E731
    for begin in range(15 * PAGE, 25 * PAGE, 1024):
        for size in (4, 1024, PAGE, PAGE + 4, 3 * PAGE, 5 * PAGE, 8 * PAGE):
            got = lib(*_query(ranges, begin), size)
            if got:
                assert all(locked(p) for p in (begin, begin + size - 1)) and all(
                    locked(p) for p in range(begin, begin + size, 1024))
            inside = any(s <= begin and begin + size <= s + n for s, n in ranges)
            assert bool(got) == inside, (begin, size)


def test_across_a_hole_is_refused(lib):
    ranges = [(16 * PAGE, 2 * PAGE), (20 * PAGE, PAGE)]
    begin, size = 17 * PAGE, 3 * PAGE + 8
    assert _query(ranges, begin)[0] and _query(ranges, begin + size - 4)[0]  # both ends are page-locked
    assert not lib(*_query(ranges, begin), size)


def test_unknown_and_overlong(lib):
    assert not lib(0, 0, 0, 0, 4)
    assert not lib(1, 0, 0, 0, 4)                       # no device address
    assert not lib(1, 4096, 8192, 4096, 4)              # a device address outside its range
    assert not lib(1, 4096, 4096, 64, 2 ** 64 - 4)      # no wrap-around
    assert lib(1, 4096, 4096, 64, 64) and not lib(1, 4100, 4096, 64, 64)
