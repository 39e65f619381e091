"""The first apply of a process may run under stream capture: everything that a capture forbids (allocations, pinned
ones among them) is done when the product is built."""
from __future__ import annotations

import subprocess
import sys

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

FIRST_APPLY = """
import ctypes as C, sys
sys.path.insert(0, {root!r})
import torch
import rooftop_mom_b200 as R
from rooftop_mom_b200 import _lib as L

p = R.Problem(R.Mesh({cx}, {cy}, 0.05, 0.05), 6.2)
n = p.rooftopCount()
op = R.Operator(p, product={product!r})
x = torch.randn(n, dtype=torch.complex128, device="cuda")
y = torch.zeros_like(x)
torch.cuda.synchronize()
g = torch.cuda.CUDAGraph()
with torch.cuda.graph(g):  # the strictest capture mode, torch's default
    s = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    a = (op.handle, C.c_void_p(x.data_ptr()), C.c_void_p(y.data_ptr()), n, 1)
    if {scratch}:
        L.call("rtm_operator_apply_fixed_scratch", *a, s)
    else:
        L.call("rtm_operator_apply", *a, L.DEVICE, s)
g.replay()
torch.cuda.synchronize()
z = op.apply(x)  # the same kernels on the same working grid size
assert torch.equal(y, z), float((y - z).abs().max())
"""


@pytest.mark.parametrize(
    "product,count,scratch",
    [("splitFFT", (100, 72), False), ("splitFFT", (64, 64), True), ("fft", (33, 28), False)],
)
def test_the_first_apply_of_a_process_can_be_captured(product, count, scratch):
    code = FIRST_APPLY.format(root=ROOT, cx=count[0], cy=count[1], product=product, scratch=scratch)
    done = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300)
    assert done.returncode == 0, done.stderr[-2000:]
