"""Solves that end before their time: a barrier of the GMRES kernels that runs out on the device (the solve fails, the next
one succeeds; tests/c/arnoldi_timeout.cu, compiled here, since the limit is internal to the library), and a cancel."""
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


def test_a_running_strip_is_cancelled_between_its_host_checks():
    """COCG on a strip looks for a cancel every 16 iterations, as on plates: a solve whose tolerance is never met stops at a
    multiple of 16 soon after the cancel, not at the end of a launch of hundreds of iterations."""
    import math
    import time

    import rooftop_mom_b200 as R

    def request():
        return R.Request.deltaGap(1501, 1, 0.05, 0.05, 2 * math.pi, method="cg", preconditioner=None, tolerance=1e-290,
                                  maxIterationCount=200000)

    stopped = []
    with R.Server(maxActive=1) as srv:
        for wait in (0.003, 0.005, 0.008, 0.003, 0.005, 0.008):
            rid = srv.submit(request())
            while srv.poll(rid)["state"] == "queued":
                time.sleep(0.0005)
            time.sleep(wait)
            srv.cancel(rid)
            done = srv.wait(rid)
            if done["state"] == "cancelled" and done["iterations"] > 0:
                stopped.append(done["iterations"])
    assert any(n % 16 == 0 and n % 512 != 0 for n in stopped), stopped
