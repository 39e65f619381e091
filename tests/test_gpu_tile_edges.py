"""Kernels at the edges of their tiles and dispatch rules, against the oracle.

Tolerances are those of the paths' parity tests: FP64 products and preconditioners 1e-13 (1e-11 for circulants,
whose spectra are divided), FP32 2e-5 (5e-6 for the block-Jacobi apply)."""
from __future__ import annotations

import math

import pytest

from conftest import random_vector, rel

pytestmark = pytest.mark.gpu

K = 2 * math.pi


def _setup(cx, cy, a=0.07, b=0.05):
    """A problem at low quadrature orders with the oracle's rooftops and the device's own generators."""
    import rooftop_mom_b200 as R
    from oracle import assembly as A, geometry as G

    prob = R.Problem(R.Mesh(cx, cy, a, b), K, quadratureOrder=(3, 3))
    xx, yy, e = prob.generators().arrays()
    rt = G.Rooftops(cx, cy, a, b, 3)
    return R, prob, rt, A.Generators(xx, yy, e, rt.content)


@pytest.mark.parametrize("precision", ["double", "single"])
@pytest.mark.parametrize("shape", [(2, 1, 2, 2), (2, 2, 2, 2), (3, 3, 2, 2), (4, 4, 1, 1), (3, 5, 8, 1), (9, 4, 2, 4),
                                   (5, 9, 1, 3), (40, 3, 3, 1), (1, 7, 2, 2), (66, 35, 2, 2)])
def test_block_jacobi_of_every_block_class(shape, precision):
    """Plates of one block, of a last column or row alone, blocks longer than the plate, and blocks whose
    unknowns do not divide a warp."""
    from oracle import blockjacobi as BJ

    cx, cy, bx, by = shape
    R, prob, rt, gen = _setup(cx, cy)
    pc = R.Preconditioner.blockJacobi(prob, (bx, by), precision=precision)
    v = random_vector(2 * rt.count, seed=3)
    got = pc.apply(v, nrhs=2)
    want = BJ.BlockJacobi(gen, rt, bx, by)
    for k in range(2):
        part = slice(k * rt.count, (k + 1) * rt.count)
        assert rel(got[part], want.apply(v[part])) < (1e-13 if precision == "double" else 5e-6)
