"""Split products on transform lengths that take every codelet of the register-resident kernels (grid_reg.cu, gen_reg.cu),
along x and along y, against the oracle. A larger transform grid gives the same product up to rounding, so any length can be
imposed on a plate of as many faces. test_host_runtime.py checks that the lengths reach every case."""
from __future__ import annotations

import math

import pytest

from conftest import random_vector, rel

# with a split of their own, and as Bluestein convolutions
LENGTHS = [12, 15, 20, 30, 42, 56, 72, 90, 120, 125, 147, 162, 168, 200, 210, 240, 256, 324, 384, 392, 405, 576, 630, 640,
           784, 875, 900, 972, 1024,
           17, 19, 26, 33, 46, 61, 65, 69, 71, 73, 99, 106, 109, 113, 127, 129, 193, 197, 241, 253, 285, 314, 385, 433, 449,
           481, 505]


@pytest.fixture(autouse=True)
def _forget_sizes():
    yield
    import rooftop_mom_b200 as R

    R.clearTuning()


@pytest.mark.gpu
@pytest.mark.parametrize("length", LENGTHS)
def test_split_products_on_imposed_lengths(length):
    import rooftop_mom_b200 as R
    from oracle import assembly as A, geometry as G, spectra as S

    for cx, cy in ((length, 18), (18, length)):
        mesh = R.Mesh(cx, cy, 0.05, 0.04)
        prob = R.Problem(mesh, 2 * math.pi, quadratureOrder=3)
        xx, yy, e = prob.generators().arrays()
        rt = G.Rooftops(cx, cy, 0.05, 0.04, 3)
        sub = S.subband_spectra(A.Generators(xx, yy, e, rt.content), 0.05, 0.04)
        v = random_vector(rt.count, seed=length)
        want = S.split_apply(rt, sub, rt.content, v)
        for precision, tolerance in (("double", 1e-13), ("single", 2e-5)):  # those of the products' other tests
            R.setTransformSize(mesh, (cx, cy), precision=precision)
            op = R.Operator(prob, precision=precision)
            assert (op.info()["fft_x"], op.info()["fft_y"]) == (cx, cy)
            assert rel(op.apply(v), want) < tolerance
            if R.fast_fft_size(length) == length:  # one y subband at a time
                lean = R.Operator(prob, product="leanSplitFFT", precision=precision)
                assert rel(lean.apply(v), want) < tolerance
