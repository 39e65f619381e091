"""A barrier of the GMRES kernels that runs out on the device ends the solve with an error, and the next solve on the
device succeeds (tests/c/arnoldi_timeout.cu, compiled here: the limit is internal to the library)."""
from __future__ import annotations

import os
import subprocess

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu


def test_a_barrier_that_runs_out_fails_the_solve_alone(tmp_path):
    from rooftop_mom_b200 import _lib as L, build

    exe = str(tmp_path / "arnoldi_timeout")
    csrc = build.CSRC
    subprocess.run([build._nvcc(), *build.ARCH, "-std=c++17", "-O2", "-w", os.path.join(ROOT, "tests", "c", "arnoldi_timeout.cu"),
                    os.path.join(csrc, "runtime.cpp"), os.path.join(csrc, "fault.cu"), "-o", exe], check=True,
                   capture_output=True, text=True)
    out = subprocess.run([exe], check=True, capture_output=True, text=True, timeout=120).stdout
    lines = {line.split()[0]: line.split()[1:] for line in out.splitlines()}
    assert lines["unpolled"][0] == str(L.ERR_TIMEOUT), out
    assert lines["default"][:2] == ["0", "1"] and float(lines["default"][2]) < 1.001e-10, out  # the monitored one is below 1e-10
