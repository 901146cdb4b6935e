"""Nothing runs beside a timed sweep.

A captured step has parallel branches; the solid's first deformation is on one that
is joined only after the sweep.  fsim_time_sweep reports the sweep's own time, so
its capture joins every branch first (launch_joins in fsim_types.h, compiled for the
CPU; that the capture asks it is read from the source).
"""
import ctypes as C
import os
import re
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "fluidsim_gb300", "csrc")
WRAPPER = """
#include "fsim_types.h"
using namespace fsim_rt;
extern "C" unsigned joins(int sweep, unsigned join, int timed)
{
    Launch L;
    L.kind = sweep ? L_SWEEP : L_VIRT;
    L.join = join;
    return launch_joins(L, timed != 0);
}
extern "C" int branches() { return kBranches; }
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("joins")
    src, so = str(d / "joins.cu"), str(d / "joins.so")
    with open(src, "w") as f:
        f.write(WRAPPER)
    subprocess.check_call(["nvcc", "-gencode", "arch=compute_103a,code=sm_103a", "-std=c++17", "-shared", "-Xcompiler",
                           "-fPIC", "-I", CSRC, src, "-o", so])
    return C.CDLL(so)


def test_a_timed_sweep_waits_for_every_branch(lib):
    every = (1 << lib.branches()) - 1
    for join in range(every + 1):
        assert lib.joins(1, join, 1) & every == every
        assert lib.joins(1, join, 0) & every == join
        for timed in (0, 1):
            assert lib.joins(0, join, timed) & every == join


def test_the_capture_joins_before_the_sweep_event():
    with open(os.path.join(CSRC, "fsim_kernels.cu")) as f:
        text = re.sub(r"//[^\n]*", "", f.read())
    body = text[text.index("fsim_status enqueue_plan("):]
    join, event = body.index("join(launch_joins(L, sweep0 != nullptr))"), body.index("cudaEventRecordWithFlags(sweep0")
    assert join < event
    assert not re.search(r"\bjoin\(L\.join\)", body)
