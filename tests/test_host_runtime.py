"""The library's host runtime (runtime.cpp, fault.cu) compiled against a stand-in for the CUDA runtime
(tests/c/host_runtime.cpp), so that what it allocates, copies and reports is checked without a GPU."""
from __future__ import annotations

import os
import shutil
import subprocess

import pytest

from conftest import ROOT


@pytest.fixture(scope="module")
def run(tmp_path_factory):
    from rooftop_mom_b200 import build

    if shutil.which("g++") is None:
        pytest.skip("no C++ compiler")
    exe = str(tmp_path_factory.mktemp("c") / "host_runtime")
    cuda = os.path.join(os.path.dirname(os.path.dirname(build._nvcc())), "include")
    subprocess.run(["g++", "-std=c++17", "-O2", "-I", cuda, "-x", "c++", os.path.join(ROOT, "tests", "c", "host_runtime.cpp"),
                    os.path.join(build.CSRC, "runtime.cpp"), os.path.join(build.CSRC, "fault.cu"), "-o", exe], check=True,
                   capture_output=True, text=True)

    def go(*args):
        out = subprocess.run([exe, *args], check=True, capture_output=True, text=True, timeout=120).stdout
        return {line.split()[0]: line.split()[1:] for line in out.splitlines()}

    return go


def test_a_fault_is_reported_by_its_own_operator(run):
    from rooftop_mom_b200 import _lib as L

    got = run("faults")
    assert got["other"] == ["0"]
    assert got["own"] == [str(L.ERR_TIMEOUT)]
    assert got["again"] == ["0"]
    assert got["reused"] == ["0", "pages", "1"]


def test_memory_that_others_take_is_refused_at_once(run):
    """A request that fitted is refused when another user of the device has taken the memory meanwhile: by the check
    itself where nothing is allocated after it (rtm_budget_require), else at the latest by the allocation."""
    from rooftop_mom_b200 import _lib as L

    got = run("budget")
    assert got["first"] == ["0"]
    assert got["taken"] == [str(L.ERR_OOM_BUDGET)]
    assert got["allocated"] == [str(L.ERR_OOM_BUDGET)]


@pytest.mark.parametrize(
    "n,kind",  # Bluestein in the Stockham engine; on register-resident lines (-1: none); sets of reordered twiddles
    [(1, (0, -1, 0)), (12, (0, 0, 0)), (13, (0, -1, 0)), (22, (0, 1, 0)), (32, (0, 0, 1)), (67, (1, 1, 0)), (97, (1, 1, 0)),
     (128, (0, 0, 1)), (256, (0, 0, 2)), (499, (1, 1, 0)), (509, (1, 1, 0)), (521, (1, -1, 0)), (1000, (0, -1, 0)),
     (1024, (0, 0, 2))],
)
def test_the_tables_of_a_length_take_one_allocation_and_one_copy(run, n, kind):
    """A set-up at a length new to the process pays for its tables: one device allocation, one copy, and entries within
    their rounding (half a unit in the last place of each part, 2^-53 sqrt(2) and 2^-24 sqrt(2), relative to the table's
    largest entry; FP32 entries are rounded twice)."""
    got = run("tables", str(n))
    assert got["cost"] == ["0", "1", "1"]
    assert tuple(int(v) for v in got["kind"]) == kind
    e64, e32 = (float(v) for v in got["errors"])
    assert e64 <= 1.01 * 2**-53 * 2**0.5
    assert e32 <= 1.01 * 2**-24 * 2**0.5


def test_the_codelet_lengths_reach_every_case_of_the_splits(run):
    """test_gpu_codelets.LENGTHS take every first and second factor that any length up to 1024 has, by register class
    (first factors up to 16, or above), with and without a Bluestein convolution: each is a case of its own in the
    kernels' switches."""
    from test_gpu_codelets import LENGTHS

    def cases(n):
        n1, n2, m = (int(v) for v in splits[str(n)])
        return {(m != n, n1 > 16, "first", n1), (m != n, n1 > 16, "second", n2)}

    splits = run("splits")
    assert len(splits) > 500
    every = set().union(*(cases(int(n)) for n in splits))
    assert set().union(*(cases(n) for n in LENGTHS)) == every
    assert min(int(n) for n in splits) in LENGTHS and max(int(n) for n in splits) in LENGTHS
