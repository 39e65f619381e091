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


# transform lengths whose splits n1 x n2 take every codelet at least once, and the smallest and largest lengths
SPLIT_GRIDS = [(16, 18), (20, 21), (24, 25), (27, 28), (30, 35), (36, 45), (49, 54), (60, 63), (75, 81), (98, 105),
               (120, 125), (126, 147), (162, 175), (196, 216), (225, 243), (250, 17), (17, 270), (288, 19), (20, 315),
               (350, 16), (16, 378), (405, 16), (18, 441), (450, 16), (16, 486), (490, 16), (16, 567), (600, 17),
               (17, 640), (700, 16), (16, 756), (840, 16), (16, 875), (945, 16), (972, 16), (16, 1008), (343, 16)]


@pytest.mark.parametrize("grid", SPLIT_GRIDS)
@pytest.mark.parametrize("precision,product", [("double", "splitFFT"), ("single", "splitFFT"),
                                               ("double", "leanSplitFFT")])
def test_split_products_of_every_codelet(grid, precision, product):
    """Face counts one below a transform length (a last column and row of padding) and the length itself."""
    from oracle import spectra as S

    for cx, cy in (grid, (grid[0] - 1, grid[1])):
        R, prob, rt, gen = _setup(cx, cy)
        v = random_vector(rt.count, seed=5)
        want = S.split_apply(rt, S.subband_spectra(gen, rt.size_x, rt.size_y), rt.content, v)
        got = R.Operator(prob, product=product, precision=precision).apply(v)
        assert rel(got, want) < (1e-13 if precision == "double" else 2e-5)


@pytest.mark.parametrize("grid", [(9, 10), (16, 17), (19, 22), (23, 18), (26, 31), (33, 37), (34, 20), (67, 61), (127, 18),
                                  (131, 16), (18, 257), (503, 17), (17, 512), (511, 19), (514, 18), (64, 48)])
@pytest.mark.parametrize("precision", ["double", "single"])
def test_circulants_of_any_face_count(grid, precision):
    """Splits, Bluestein convolutions up to their longest (512) and lengths beyond the register-resident form, for
    one vector and for three; the embedding product (periods 2 n - 2) on the smaller grids."""
    from oracle import preconditioner as Q, spectra as S

    R, prob, rt, gen = _setup(*grid)
    v = random_vector(3 * rt.count, seed=6)
    spec = Q.circulant(gen, rt.size_x, rt.size_y, kernel="rChan")
    pc = R.Preconditioner(prob, kernel="rChan", precision=precision)
    got, one = pc.apply(v, nrhs=3), pc.apply(v[:rt.count])
    for k in range(3):
        part = slice(k * rt.count, (k + 1) * rt.count)
        assert rel(got[part], S.fft_apply(rt, spec, rt.content, v[part])) < (1e-11 if precision == "double" else 2e-5)
    assert rel(one, got[:rt.count]) < 1e-15
    if max(grid) <= 67:
        emb = S.embedding_spectra(gen, rt.size_x, rt.size_y)
        want = S.fft_apply(rt, emb, rt.content, v[:rt.count])
        got = R.Operator(prob, product="fft", precision=precision).apply(v[:rt.count])
        assert rel(got, want) < (1e-13 if precision == "double" else 2e-5)


@pytest.mark.parametrize("count", [(2, 1), (3, 1), (17, 1), (1, 40), (134, 1), (400, 1), (1, 701), (1600, 1)])
@pytest.mark.parametrize("preconditioned", [True, False])
def test_strip_solves(count, preconditioned):
    """COCG on strips from the shortest to one that fits a CTA without the circulant alone, three right-hand sides at
    once, one of them zero, and from an initial guess. The recurrence's history hangs on rounding past its first
    iterations (the oracle's own moves by 0.5 % when b moves by 1e-15), so what is checked is what does not: the first
    residuals, the iteration counts at 1e-6 (within 2, as for plates), and the residual of the returned current through
    the oracle's product against the reported one."""
    import numpy as np

    from oracle import preconditioner as Q, solvers, spectra as S

    R, prob, rt, gen = _setup(*count, a=0.05, b=0.05)
    sub = S.subband_spectra(gen, rt.size_x, rt.size_y)
    A = lambda v: S.split_apply(rt, sub, rt.content, v)  # noqa: E731
    op, pc, M = R.Operator(prob, maxRhs=3), None, None
    if preconditioned:
        pc = R.Preconditioner(prob, kernel="rChan")
        spec = Q.circulant(gen, rt.size_x, rt.size_y, kernel="rChan")
        M = lambda v: S.fft_apply(rt, spec, rt.content, v)  # noqa: E731
    n = rt.count
    b = np.concatenate([random_vector(n, seed=1), np.zeros(n), random_vector(n, seed=2)])
    limit = 60 if preconditioned or n == 1 else 3
    solver = R.Solver("cg", tolerance=1e-6, maxIterationCount=limit)
    got = solver.solve(op, b, preconditioner=pc, nrhs=3)
    for k, r in enumerate(got):
        part = b[k * n:(k + 1) * n]
        if k == 1:
            assert r.converged() and r.iterationCount() == 0 and not np.any(r.solution()) and r.residualNorm() == 0
            continue
        want = solvers.solve("cg", A, part, tol=1e-6, maxit=limit, precond=M)
        assert r.converged() == want.converged and abs(r.iterationCount() - want.iteration_count) <= 2
        assert len(r.residualNorms()) == r.iterationCount() + 1
        assert np.allclose(r.residualNorms()[:3], want.residual_norms[:3], rtol=1e-9)
        true = np.linalg.norm(part - A(r.solution())) / np.linalg.norm(part)
        assert abs(r.residualNorm() - true) < 1e-10
        assert not r.converged() or true < 1e-5
    again = solver.solve(op, b[:n], preconditioner=pc, initialGuess=got[0].solution())
    assert abs(again.residualNorms()[0] - got[0].residualNorm()) < 1e-10


def test_a_strip_solve_of_more_iterations_than_one_launch():
    """An unreachable tolerance runs to the iteration limit over several launches of the strip kernel."""
    import numpy as np

    R, prob, rt, gen = _setup(500, 1, a=0.05, b=0.05)
    op = R.Operator(prob)
    res = R.Solver("cg", tolerance=1e-300, maxIterationCount=1100).solve(op, random_vector(rt.count, seed=4))
    assert not res.converged() and res.iterationCount() in range(1, 1101)
    assert len(res.residualNorms()) == res.iterationCount() + 1
    # the recurrence either ran out or broke down to a value that is not finite
    assert res.iterationCount() == 1100 or not np.isfinite(res.residualNorms()[-1])


def _gmres_case(n, seed, nrhs):
    import numpy as np

    rng = np.random.default_rng(seed)
    A = np.eye(n) + 0.4 * (rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))) / math.sqrt(2 * n)
    return A, random_vector(n * nrhs, seed=seed + 1)


@pytest.mark.parametrize("n,restart,nrhs", [(1, 1, 1), (2, 5, 1), (31, 15, 2), (33, 16, 3), (129, 17, 1), (130, 32, 5),
                                            (257, 33, 1), (300, 63, 1), (300, 64, 1), (700, 50, 2), (40, 20, 75)])
@pytest.mark.parametrize("passes", [2, 1])
def test_arnoldi_steps(n, restart, nrhs, passes):
    """GMRES over bases from one column to the longest of the one-launch Arnoldi step (63) and one beyond it, rows from
    one to several CTAs, and right-hand sides from one to more than a device's CTAs: the oracle's residual histories
    (its orthogonalisation is backward stable, so they agree to a few roundings: 1e-8) and solutions."""
    import numpy as np

    import rooftop_mom_b200 as R
    from oracle import solvers

    A, b = _gmres_case(n, 11, nrhs)
    solver = R.Solver("gmres", tolerance=1e-10, maxIterationCount=90, restart=restart, gramSchmidtPasses=passes)
    got = solver.solve(R.DenseOperator(A), b, nrhs=nrhs)
    for k, r in enumerate(got if nrhs > 1 else [got]):
        want = solvers.solve("gmres", A, b[k * n:(k + 1) * n], tol=1e-10, maxit=90, restart=restart)
        assert r.converged() == want.converged and abs(r.iterationCount() - want.iteration_count) <= 1
        h = min(r.iterationCount(), want.iteration_count) + 1
        assert np.allclose(r.residualNorms()[:h], want.residual_norms[:h], rtol=1e-8, atol=1e-13)
        assert rel(r.solution(), want.solution) < 1e-8


def test_arnoldi_steps_whose_basis_spans_the_solution():
    """A matrix whose Krylov space ends after three steps: the second projection removes all there is, so the norm is
    summed rather than subtracted, and the solve ends there."""
    import numpy as np

    import rooftop_mom_b200 as R

    n = 500
    rng = np.random.default_rng(5)
    u = np.linalg.qr(rng.standard_normal((n, 2)) + 1j * rng.standard_normal((n, 2)))[0]
    A = np.eye(n) + u @ np.diag([2.0, 5.0j]) @ u.conj().T
    b = random_vector(n, seed=9)
    res = R.Solver("gmres", tolerance=1e-12, maxIterationCount=40, restart=20).solve(R.DenseOperator(A), b)
    assert res.converged() and res.iterationCount() == 3
    assert rel(A @ res.solution(), b) < 1e-12


@pytest.mark.parametrize("grid", [(1, 2), (2, 1), (2, 2), (3, 7), (7, 3), (31, 33), (40, 40), (64, 5), (5, 64), (90, 1)])
@pytest.mark.parametrize("sizes,orders", [((0.05, 0.05), (16, 8)), ((0.05, 0.05), (4, 1)), ((0.07, 0.05), (5, 3)),
                                          ((0.05, 0.05), (6, 33)), ((0.02, 0.05), (4, 5))])
def test_assembled_generators(grid, sizes, orders):
    """Square faces (half the far blocks evaluated, the others mirrored) and others, grids wider and taller than the
    triangle of mirrored blocks, and rules from one point to more rows than a pass takes: the oracle's generators to
    1e-12 in norm."""
    import rooftop_mom_b200 as R
    from oracle import assembly as A

    prob = R.Problem(R.Mesh(*grid, *sizes), K, quadratureOrder=orders)
    got = prob.generators().arrays()
    want = A.generate(*grid, *sizes, K, orders)
    for g, w in zip(got, (want.magnetic_xx, want.magnetic_yy, want.electric)):
        if w is not None and w.size:
            assert rel(g, w) < 1e-12


@pytest.mark.parametrize("grid", [(256, 33), (33, 256), (255, 35), (512, 21), (19, 511), (256, 256), (1024, 18), (17, 1023)])
@pytest.mark.parametrize("precision", ["double", "single"])
def test_lines_of_three_steps(grid, precision):
    """Transform lengths 256, 512 and 1024 along either direction or both, beside lengths of the register-resident form
    and an odd number of lines; a last row of padding; one vector and three. The split product, the circulant, and the
    embedding whose period 2 n - 2 is 256."""
    from oracle import preconditioner as Q, spectra as S

    R, prob, rt, gen = _setup(*grid)
    v = random_vector(3 * rt.count, seed=9)
    sub = S.subband_spectra(gen, rt.size_x, rt.size_y)
    circ = Q.circulant(gen, rt.size_x, rt.size_y, kernel="rChan")
    op, pc = R.Operator(prob, precision=precision, maxRhs=3), R.Preconditioner(prob, kernel="rChan", precision=precision)
    got, pre = op.apply(v, nrhs=3), pc.apply(v, nrhs=3)
    for k in range(3):
        part = slice(k * rt.count, (k + 1) * rt.count)
        assert rel(got[part], S.split_apply(rt, sub, rt.content, v[part])) < (1e-13 if precision == "double" else 2e-5)
        assert rel(pre[part], S.fft_apply(rt, circ, rt.content, v[part])) < (1e-11 if precision == "double" else 2e-5)
    assert rel(op.apply(v[:rt.count]), got[:rt.count]) < 1e-15
    if grid == (33, 256):
        R, prob, rt, gen = _setup(129, grid[0])
        emb = S.embedding_spectra(gen, rt.size_x, rt.size_y)
        got = R.Operator(prob, product="fft", precision=precision).apply(v[:rt.count])
        assert rel(got, S.fft_apply(rt, emb, rt.content, v[:rt.count])) < (1e-13 if precision == "double" else 2e-5)


@pytest.mark.parametrize("grid", [(2, 2), (16, 17), (16, 18), (23, 23), (45, 46), (46, 46), (64, 65), (65, 65), (91, 91),
                                  (91, 92)])
@pytest.mark.parametrize("preconditioned", [True, False])
def test_cocg_steps_by_row_chunks(grid, preconditioned):
    """One chunk of rows to one more than a cluster takes, and the first size above: the residuals of five iterations,
    which rounding has not yet moved, for two systems and a zero one, and the current they leave."""
    import numpy as np

    from oracle import preconditioner as Q, solvers, spectra as S

    R, prob, rt, gen = _setup(*grid)
    sub = S.subband_spectra(gen, rt.size_x, rt.size_y)
    A = lambda v: S.split_apply(rt, sub, rt.content, v)  # noqa: E731
    pc = M = None
    if preconditioned:
        pc = R.Preconditioner(prob, kernel="rChan")
        spec = Q.circulant(gen, rt.size_x, rt.size_y, kernel="rChan")
        M = lambda v: S.fft_apply(rt, spec, rt.content, v)  # noqa: E731
    n = rt.count
    limit = min(5, n)
    b = np.concatenate([random_vector(n, seed=3), np.zeros(n), random_vector(n, seed=4)])
    got = R.Solver("cg", tolerance=1e-14, maxIterationCount=limit).solve(R.Operator(prob, maxRhs=3), b, preconditioner=pc,
                                                                       nrhs=3)
    for k, r in enumerate(got):
        if k == 1:
            assert r.converged() and r.iterationCount() == 0 and not np.any(r.solution())
            continue
        want = solvers.solve("cg", A, b[k * n:(k + 1) * n], tol=1e-14, maxit=limit, precond=M)
        count = min(r.iterationCount(), want.iteration_count) + 1
        above = want.residual_norms[:count] > 1e-10  # the smallest system converges within the limit
        assert above[0] and np.allclose(r.residualNorms()[:count][above], want.residual_norms[:count][above], rtol=1e-9)
        true = np.linalg.norm(b[k * n:(k + 1) * n] - A(r.solution())) / np.linalg.norm(b[k * n:(k + 1) * n])
        assert abs(true - r.residualNorm()) < 1e-10
