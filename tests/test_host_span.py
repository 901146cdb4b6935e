"""The rule by which a kernel may copy to and from a caller's host buffer itself
(fluidsim_gb300/csrc/fsim_span.h), compiled for the CPU.

A buffer may begin in one page-locked allocation and end in another with pages in
between that the device cannot reach, so both ends being page-locked is not
enough.  Such a buffer is never handed to the GPU here.
"""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from fluidsim_gb300 import api, cases

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "fluidsim_gb300", "csrc")
WRAPPER = """
#include "fsim_span.h"
extern "C" int addressable(int host, uintptr_t dev, uintptr_t start, size_t size, size_t bytes)
{
    return fsim_rt::span_addressable({host != 0, dev, start, size}, bytes);
}
extern "C" int overlap(uintptr_t p, size_t n, uintptr_t q, size_t m) { return fsim_rt::spans_overlap(p, n, q, m); }
"""
PAGE = 4096


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("span")
    src, so = str(d / "span.cpp"), str(d / "span.so")
    with open(src, "w") as f:
        f.write(WRAPPER)
    subprocess.check_call(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-I", CSRC, src, "-o", so])
    so = C.CDLL(so)
    so.addressable.argtypes = [C.c_int, C.c_size_t, C.c_size_t, C.c_size_t, C.c_size_t]
    so.overlap.argtypes = [C.c_size_t] * 4
    return so


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
            got = lib.addressable(*_query(ranges, begin), size)
            if got:
                assert all(locked(p) for p in (begin, begin + size - 1)) and all(
                    locked(p) for p in range(begin, begin + size, 1024))
            inside = any(s <= begin and begin + size <= s + n for s, n in ranges)
            assert bool(got) == inside, (begin, size)


def test_across_a_hole_is_refused(lib):
    ranges = [(16 * PAGE, 2 * PAGE), (20 * PAGE, PAGE)]
    begin, size = 17 * PAGE, 3 * PAGE + 8
    assert _query(ranges, begin)[0] and _query(ranges, begin + size - 4)[0]  # both ends are page-locked
    assert not lib.addressable(*_query(ranges, begin), size)


def test_unknown_and_overlong(lib):
    assert not lib.addressable(0, 0, 0, 0, 4)
    assert not lib.addressable(1, 0, 0, 0, 4)                       # no device address
    assert not lib.addressable(1, 4096, 8192, 4096, 4)              # a device address outside its range
    assert not lib.addressable(1, 4096, 4096, 64, 2 ** 64 - 4)      # no wrap-around
    assert lib.addressable(1, 4096, 4096, 64, 64) and not lib.addressable(1, 4100, 4096, 64, 64)


def test_overlap_against_the_bytes(lib):
    for p in range(8, 14):
        for q in range(8, 14):
            for n in range(0, 5):
                for m in range(0, 5):
                    assert bool(lib.overlap(p, n, q, m)) == bool(set(range(p, p + n)) & set(range(q, q + m)))


@pytest.mark.gpu
def test_last_field_wins_in_a_shared_buffer():
    """Fields read into one buffer leave the last one's bytes, whichever kind of memory it is."""
    cfg, pa = cases.make(cases.tiny_box(jitter=0.01))
    names = ("fluid_pos", "fluid_vel")
    rng = np.random.default_rng(1)
    with api.Simulation(cfg, pa, device=0) as sim:
        sim.set("fluid_vel", rng.uniform(-1, 1, pa.fluid_vel.shape).astype(np.float32))
        n = pa.fluid_vel.nbytes
        for order in (names, names[::-1]):
            for shift in (0, 64):
                # the first field's buffer `shift` bytes in (the buffer is longer by as much)
                owner = api.PinnedBuffer((n + 64,), np.uint8)
                p = owner.array.ctypes.data
                sim.get_many_ptr(order, [p + shift, p], [n, n])
                assert owner.array[:n].tobytes() == sim.get(order[1]).tobytes()
                assert owner.array[n:n + shift].tobytes() == sim.get(order[0]).tobytes()[n - shift:n]
