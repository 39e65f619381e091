"""The work a user of this framework has it do, as measurable cases over its public API.

A user meets the framework in four ways, and the cases stand for these:

- products and preconditioners applied to vectors on the device (every iteration of every solve);
- the set-up of a new plate or a new frequency: assembly, product, preconditioner, plane wave, first applies;
- solves of one plate, one right-hand side or several, as far as a fixed number of iterations, so that two
  builds do the same work; strips fed by a delta gap among them;
- plates of uneven size solved together.

Sizes are those of the benchmark's workloads (32 x 32, 256 x 256, 512 x 512 and 1024 x 1024 plates; 33 to 64
faces a side for the uneven plates; 16 to 768 faces a side, half of them strips, for the request stream), with
cells of 1/10 to 1/25 wavelength. Inputs are generators assembled by the framework, plane waves and random
vectors, all made from the seed.

exact() restates the same quantities in 64 bits: the moments by Gauss-Legendre rules of higher orders (the
singular ones in Duffy's coordinates), the Toeplitz products through a 2n x 2n embedding, the solvers by their
definitions, on plain torch tensors.
"""
from __future__ import annotations

import cmath
import functools
import math

import numpy as np
import torch

import rooftop_mom_b200 as R

Z0 = 376.730313668  # ohm, the framework's constant


def listed():
    return [
        # the smallest plate of the benchmark: one product, where launches and the call itself count
        {"name": "product_32", "kind": "product", "cx": 32, "cy": 32, "product": "splitFFT",
         "precision": "double", "rhs": 1, "density": 20.0},
        # the benchmark's headline plate: its product in double precision
        {"name": "product_256", "kind": "product", "cx": 256, "cy": 256, "product": "splitFFT",
         "precision": "double", "rhs": 1, "density": 20.0},
        # a plate as a mesher leaves it: uneven and odd face counts (transforms of 315 x 189 points)
        {"name": "product_301x187", "kind": "product", "cx": 301, "cy": 187, "product": "splitFFT",
         "precision": "double", "rhs": 1, "density": 17.0},
        # the largest plate of the benchmark, in the single precision of its inner iterations
        {"name": "product_1024_single", "kind": "product", "cx": 1024, "cy": 1024, "product": "splitFFT",
         "precision": "single", "rhs": 1, "density": 15.0},
        # the default preconditioner on the batching workload's plate, some right-hand sides at once
        {"name": "circulant_512_rhs4", "kind": "circulant", "cx": 512, "cy": 512, "kernel": "rChan",
         "precision": "double", "rhs": 4, "density": 20.0},
        # a new frequency on the headline plate: everything before its solve, and the first applies
        {"name": "setup_256_blockJacobi", "kind": "setup", "cx": 256, "cy": 256, "pc": "blockJacobi",
         "density": 20.0},
        # the same for a plate of the request stream, with the default preconditioner
        {"name": "setup_250x139_rChan", "kind": "setup", "cx": 250, "cy": 139, "pc": "rChan", "density": 14.0},
        # the headline solve, two restart cycles of it: block-Jacobi GMRES(50), one plane wave
        {"name": "gmres_256", "kind": "solve", "cx": 256, "cy": 256, "method": "gmres", "pc": "blockJacobi",
         "side": "right", "rhs": 1, "iterations": 100, "density": 20.0},
        # the smallest solve: COCG without a preconditioner
        {"name": "cocg_32", "kind": "solve", "cx": 32, "cy": 32, "method": "cg", "pc": "none", "side": "left",
         "rhs": 1, "iterations": 32, "density": 20.0},
        # the batching workload: several plane waves at once on a large plate, rChan COCG (the recurrence
        # amplifies rounding, so that two builds stay comparable for its first iterations alone)
        {"name": "cocg_512_rhs8", "kind": "solve", "cx": 512, "cy": 512, "method": "cg", "pc": "rChan",
         "side": "left", "rhs": 8, "iterations": 12, "density": 20.0},
        # half of the request stream: a strip fed by a delta gap, solved to 1e-6, with its impedance
        {"name": "strip_400", "kind": "strip", "cx": 400, "density": 18.0},
        # plates of uneven size solved as one batch, one restart cycle
        {"name": "uneven_16", "kind": "uneven", "plates": 16, "low": 33, "high": 64, "layout": 0,
         "iterations": 50, "density": 20.0},
    ]


def _log_int(rng, low, high):
    return max(low, min(high, int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))))


def draw(rng):
    kind = rng.choice(["product"] * 5 + ["circulant"] * 2 + ["setup"] + ["solve"] * 3 + ["strip"] + ["uneven"])
    density = round(rng.uniform(10.0, 25.0), 3)
    if kind == "product":
        precision = rng.choice(["double", "double", "single"])
        product = rng.choice(["splitFFT"] * 4 + ["leanSplitFFT", "fft"])
        # the embedding product doubles the transform lengths
        high = 384 if product == "fft" else 768
        cx, cy = _log_int(rng, 16, high), _log_int(rng, 16, high)
        rhs = rng.choice([1, 1, 1, 2, 4, 8]) if cx * cy <= 100000 else 1
        return {"kind": kind, "cx": cx, "cy": cy, "product": product, "precision": precision, "rhs": rhs,
                "density": density}
    if kind == "circulant":
        cx, cy = _log_int(rng, 16, 768), _log_int(rng, 16, 768)
        rhs = rng.choice([1, 1, 2, 4, 8]) if cx * cy <= 100000 else 1
        return {"kind": kind, "cx": cx, "cy": cy, "kernel": rng.choice(["rChan", "rChan", "tChan", "strang"]),
                "precision": rng.choice(["double", "double", "single"]), "rhs": rhs, "density": density}
    if kind == "setup":
        return {"kind": kind, "cx": _log_int(rng, 16, 512), "cy": _log_int(rng, 16, 512),
                "pc": rng.choice(["blockJacobi", "rChan"]), "density": density}
    if kind == "solve":
        cx, cy = _log_int(rng, 16, 512), _log_int(rng, 16, 512)
        rhs = rng.choice([1, 1, 2, 4]) if cx * cy <= 70000 else 1
        method, pc, side = rng.choice([("gmres", "blockJacobi", "right"), ("cg", "rChan", "left"),
                                       ("gmres", "blockJacobi", "left"), ("cg", "none", "left")])
        return {"kind": kind, "cx": cx, "cy": cy, "method": method, "pc": pc, "side": side, "rhs": rhs,
                "iterations": rng.randint(20, 70) if method == "gmres" else rng.randint(8, 12),
                "density": density}
    if kind == "strip":
        return {"kind": kind, "cx": _log_int(rng, 16, 768), "density": density}
    low = rng.randint(33, 56)
    return {"kind": kind, "plates": rng.randint(4, 16), "low": low, "high": 64,
            "layout": rng.randint(1, 10**6), "iterations": rng.randint(25, 50), "density": density}


# ---------------------------------------------------------------------------------------------
# what the seed gives: the wavenumber (a frequency within a few per cent of the nominal one), waves, vectors
def _wavenumber(seed):
    return 2 * math.pi * float(np.random.default_rng(seed).uniform(0.96, 1.0))


def _waves(seed, count):
    """theta ~ U[0, 80] deg, phi ~ U[0, 360) deg, TE or TM, as the batching workload draws them."""
    rng = np.random.default_rng([seed, 1])
    waves = []
    for _ in range(count):
        t, p = math.radians(rng.uniform(0.0, 80.0)), math.radians(rng.uniform(0.0, 360.0))
        d = (math.sin(t) * math.cos(p), math.sin(t) * math.sin(p), -math.cos(t))
        te = (-math.sin(p), math.cos(p), 0.0)
        tm = (math.cos(t) * math.cos(p), math.cos(t) * math.sin(p), math.sin(t))
        waves.append((d, te if rng.random() < 0.5 else tm))
    return waves


def _vector(seed, n, precision, device):
    rng = np.random.default_rng([seed, 2])
    v = rng.standard_normal(2 * n).view(np.complex128)
    return torch.from_numpy(v).to(device, torch.complex64 if precision == "single" else torch.complex128)


def _uneven_sizes(case):
    rng = np.random.default_rng(case["layout"])
    return [(int(x), int(y)) for x, y in rng.integers(case["low"], case["high"] + 1, size=(case["plates"], 2))]


def _rooftops(cx, cy):
    return (cx - 1) * cy + cx * (cy - 1)


def _problem(cx, cy, density, seed):
    h = 1.0 / density
    return R.Problem(R.Mesh(cx, cy, h, h), _wavenumber(seed))


def _preconditioner(problem, pc):
    if pc == "none":
        return None
    return R.Preconditioner.blockJacobi(problem, (2, 2)) if pc == "blockJacobi" else R.Preconditioner(problem, pc)


def prepare(case, seed):
    kind = case["kind"]
    state = {"case": case}
    if kind in ("product", "circulant"):
        problem = _problem(case["cx"], case["cy"], case["density"], seed)
        n = _rooftops(case["cx"], case["cy"])
        if kind == "product":
            state["op"] = R.Operator(problem, product=case["product"], precision=case["precision"],
                                     maxRhs=case["rhs"])
        else:
            state["op"] = R.Preconditioner(problem, kernel=case["kernel"], precision=case["precision"])
        state["x"] = _vector(seed, n * case["rhs"], case["precision"], "cuda")
    elif kind == "setup":
        state["wavenumber"] = _wavenumber(seed)
        state["wave"] = _waves(seed, 1)[0]
        state["x"] = _vector(seed, _rooftops(case["cx"], case["cy"]), "double", "cuda")
    elif kind == "solve":
        problem = _problem(case["cx"], case["cy"], case["density"], seed)
        state["op"] = R.Operator(problem, maxRhs=case["rhs"])
        state["pc"] = _preconditioner(problem, case["pc"])
        waves = [R.Excitation.planeWave(problem, d, p, device=True) for d, p in _waves(seed, case["rhs"])]
        state["rhs"] = waves[0] if len(waves) == 1 else torch.cat([w.vector() for w in waves])
        state["solver"] = R.Solver(case["method"], tolerance=1e-13, maxIterationCount=case["iterations"],
                                   restart=50, side=case["side"])
    elif kind == "strip":
        problem = _problem(case["cx"], 1, case["density"], seed)
        state["op"] = R.Operator(problem)
        state["pc"] = R.Preconditioner(problem, "rChan")
        state["rhs"] = R.Excitation.deltaGap(problem, direction="x", voltage=1.0)
        state["solver"] = R.Solver("cg", tolerance=1e-6)
    else:
        h = 1.0 / case["density"]
        ops, pcs, rhs = [], [], []
        for (cx, cy), (d, p) in zip(_uneven_sizes(case), _waves(seed, case["plates"])):
            mesh = R.Mesh(cx, cy, h, h)
            R.setTransformSize(mesh, (64, 64))
            problem = R.Problem(mesh, _wavenumber(seed))
            ops.append(R.Operator(problem))
            pcs.append(R.Preconditioner.blockJacobi(problem, (2, 2)))
            rhs.append(R.Excitation.planeWave(problem, d, p, device=True))
        R.clearTuning()  # the operators keep their grids; other cases take the reference's
        state["batch"] = R.PlateBatch(ops, pcs)
        state["rhs"] = rhs
        state["solver"] = R.Solver("gmres", tolerance=1e-13, maxIterationCount=case["iterations"], restart=50,
                                   side="right")
    torch.cuda.synchronize()
    return state


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind in ("product", "circulant"):
        return state["op"].apply(state["x"], nrhs=case["rhs"])
    if kind == "setup":
        h = 1.0 / case["density"]
        problem = R.Problem(R.Mesh(case["cx"], case["cy"], h, h), state["wavenumber"])
        op = R.Operator(problem)
        pc = _preconditioner(problem, case["pc"])
        wave = R.Excitation.planeWave(problem, *state["wave"], device=True)
        return {"product": op.apply(state["x"]), "preconditioned": pc.apply(state["x"]), "wave": wave.vector()}
    if kind == "solve":
        result = state["solver"].solve(state["op"], state["rhs"], preconditioner=state["pc"], nrhs=case["rhs"])
        if case["rhs"] > 1:
            return {"x": [r.solution() for r in result], "history": [r.residualNorms() for r in result],
                    "iterations": [r.iterationCount() for r in result]}
        return {"x": result.solution(), "history": result.residualNorms(), "iterations": result.iterationCount(),
                "rcs": result.radarCrossSection()}
    if kind == "strip":
        result = state["solver"].solve(state["op"], state["rhs"], preconditioner=state["pc"])
        z = result.inputImpedance()
        return {"x": result.solution(), "iterations": result.iterationCount(), "impedance": [z.real, z.imag]}
    results = state["solver"].solveBatch(state["batch"], state["rhs"])
    return {"x": [r.solution() for r in results], "history": [r.residualNorms() for r in results],
            "iterations": [r.iterationCount() for r in results]}


# ---------------------------------------------------------------------------------------------
# work: inputs read once, outputs written once, and the operations of the transforms and recurrences
def _product_work(cx, cy, rhs, element):
    """The vectors and the three generators' spectra on the 2n x 2n periods (their quarter, by evenness)."""
    n, points = _rooftops(cx, cy), 4.0 * cx * cy
    flops = rhs * (4 * 5 * points * math.log2(max(2.0, points)) + 40 * points)
    return element * (2.0 * n * rhs + 3 * cx * cy), flops


def _circulant_work(cx, cy, rhs, element):
    n, points = _rooftops(cx, cy), float(cx * cy)
    return element * (2.0 * n * rhs + 3 * points), rhs * (4 * 5 * points * math.log2(max(2.0, points)) + 28 * points)


def _setup_work(cx, cy):
    """Far-lattice kernel values (64 a block) with their weights, three generators transformed and stored."""
    blocks, points = (cx + 1.0) * (cy + 1.0), 4.0 * cx * cy
    flops = blocks * 64 * (2 * 28 * 2 + 40) + 3 * 5 * points * math.log2(points)
    return 16.0 * (3 * cx * cy * 2 + 6 * _rooftops(cx, cy)), flops


def _solve_work(cx, cy, method, pc, rhs, iterations, restart=50):
    n = _rooftops(cx, cy)
    pb, pf = _product_work(cx, cy, rhs, 16)
    if pc == "rChan":
        mb, mf = _circulant_work(cx, cy, rhs, 16)
    elif pc == "blockJacobi":
        mb, mf = 16.0 * 2 * n * rhs, 8.0 * 8 * n * rhs
    else:
        mb = mf = 0.0
    if method == "cg":  # r, z, d, q, x: the recurrences' vectors read and written once an iteration
        vb, vf = 16.0 * 8 * n * rhs * iterations, 4 * 8.0 * n * rhs * iterations
    else:  # the basis read for the two projections and the two corrections
        columns = sum((i % restart) + 1 for i in range(iterations))
        vb, vf = 16.0 * n * rhs * (2 * columns + 4 * iterations), 4 * 8.0 * n * rhs * columns
    return iterations * (pb + mb) + vb, iterations * (pf + mf) + vf


def work(case):
    kind = case["kind"]
    if kind == "product":
        b, f = _product_work(case["cx"], case["cy"], case["rhs"], 8 if case["precision"] == "single" else 16)
    elif kind == "circulant":
        b, f = _circulant_work(case["cx"], case["cy"], case["rhs"], 8 if case["precision"] == "single" else 16)
    elif kind == "setup":
        b, f = _setup_work(case["cx"], case["cy"])
    elif kind == "solve":
        b, f = _solve_work(case["cx"], case["cy"], case["method"], case["pc"], case["rhs"], case["iterations"])
    elif kind == "strip":
        n, it = case["cx"] - 1.0, 6  # about what these strips take
        b, f = 16.0 * 14 * n * it, it * (6 * 5 * 2 * n * math.log2(2 * n) + 60 * n)
    else:
        side = (case["low"] + case["high"]) // 2
        b, f = _solve_work(side, side, "gmres", "blockJacobi", case["plates"], case["iterations"])
    return {"bytes": float(b), "flops": float(f)}


# ---------------------------------------------------------------------------------------------
# exact: plain torch in 64 bits. Grids are [x, y]; rooftop vectors are their column-major flattening, the
# x-directed grid first.
def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _rule(order):
    p, w = np.polynomial.legendre.leggauss(order)
    return torch.from_numpy((p + 1) / 2).to(_device()), torch.from_numpy(w / 2).to(_device())


def _axis_weights(nu):
    """The four difference-coordinate weights of two linear functions on neighbouring cells: 1 - |nu| and the
    first and mixed moments."""
    d = nu.abs()
    left = nu < 0
    w10 = torch.where(left, (1 + nu) ** 2 / 2, (1 - nu**2) / 2)
    w01 = torch.where(left, (1 - nu**2) / 2, (1 - nu) ** 2 / 2)
    return torch.stack([1 - d, w10, w01, (1 - d) ** 2 * (2 + d) / 6])


def _moments_at(nu, eta, weight, dx, dy, a, b, k):
    """The 7 moments of cell offsets (dx, dy) over the points (nu, eta) [p] with their quadrature weights."""
    wx, wy = _axis_weights(nu), _axis_weights(eta)
    w = torch.cat([wy[0] * wx, wy[1:] * wx[0]]) * weight
    r = torch.hypot(a * (nu[:, None] - dx), b * (eta[:, None] - dy))
    return w.to(torch.complex128) @ (torch.exp(-1j * k * r) / r)


def _touching(dx, dy, a, b, k, order=40):
    """The moments of an offset whose kernel is singular within the rule: per quadrant, Duffy's coordinates
    about the singular corner, or the plain rule where the corner is not the quadrant's."""
    p, w = _rule(order)
    u, v = torch.meshgrid(p, p, indexing="ij")
    uv_w = (w[:, None] * w[None, :]).reshape(-1)
    u, v = u.reshape(-1), v.reshape(-1)
    total = 0
    off = torch.tensor
    for x0 in (-1.0, 0.0):
        for y0 in (-1.0, 0.0):
            corner = dx in (x0, x0 + 1) and dy in (y0, y0 + 1)
            if not corner:
                pieces = [(u, v, uv_w)]
                sx, sy, ox, oy = 1.0, 1.0, x0, y0
            else:
                pieces = [(u, u * v, uv_w * u), (u * v, u, uv_w * u)]
                sx, sy = (1.0 if dx == x0 else -1.0), (1.0 if dy == y0 else -1.0)
                ox, oy = float(dx), float(dy)
            for s, t, ww in pieces:
                nu, eta = ox + sx * s, oy + sy * t
                total = total + _moments_at(nu, eta, ww, off([float(dx)], device=_device(), dtype=torch.float64),
                                            off([float(dy)], device=_device(), dtype=torch.float64), a, b, k)[:, 0]
    return total


def _plain(dx, dy, a, b, k, order):
    """The moments [7, offsets] of offsets away from the singularity."""
    p, w = _rule(order)
    nu1, w1 = torch.cat([p - 1, p]), torch.cat([w, w])
    nu, eta = torch.meshgrid(nu1, nu1, indexing="ij")
    ww = (w1[:, None] * w1[None, :]).reshape(-1)
    out = []
    step = max(1, 32_000_000 // nu.numel())
    for i in range(0, dx.numel(), step):
        out.append(_moments_at(nu.reshape(-1), eta.reshape(-1), ww, dx[i:i + step], dy[i:i + step], a, b, k))
    return torch.cat(out, dim=1)


@functools.lru_cache(maxsize=20)
def _generators(cx, cy, h, k):
    """The three generators E [cx, cy], XX [cx - 1, cy], YY [cx, cy - 1] of square cells of side h."""
    dev = _device()
    gx, gy = torch.meshgrid(torch.arange(cx, device=dev), torch.arange(cy, device=dev), indexing="ij")
    gx, gy = gx.reshape(-1).double(), gy.reshape(-1).double()
    moments = torch.empty(7, cx * cy, dtype=torch.complex128, device=dev)
    near = (gx < 6) & (gy < 6)
    moments[:, ~near] = _plain(gx[~near], gy[~near], h, h, k, 10)
    moments[:, near] = _plain(gx[near], gy[near], h, h, k, 32)
    for dx in range(min(2, cx)):
        for dy in range(min(2, cy)):
            moments[:, dx * cy + dy] = _touching(dx, dy, h, h, k)
    m = moments.reshape(7, cx, cy)
    scale = 1j * Z0 / (4 * math.pi) * h**4
    E = scale / k * m[0]
    t = scale * k

    def rising(dim, near_term, up, mixed):
        own = m[0] - m[near_term] - m[up] + 2 * m[mixed]
        rise, fall = m[near_term] - m[mixed], m[up] - m[mixed]
        n = m.shape[dim]
        g = own.narrow(dim - 1, 0, n - 1).clone()
        doubled = rise.narrow(dim - 1, 1, n - 1).clone()
        doubled.narrow(dim - 1, 0, min(1, n - 1)).mul_(2)
        g += doubled
        if n > 2:
            g.narrow(dim - 1, 1, n - 2).add_(fall.narrow(dim - 1, 0, n - 2))
        return t * g

    return E, rising(1, 1, 2, 3), rising(2, 4, 5, 6)


def _split(x, cx, cy):
    """[rhs, n] vectors as the two grids [rhs, x, y]."""
    nx, rhs = (cx - 1) * cy, x.shape[0]
    return (x[:, :nx].reshape(rhs, cy, cx - 1).transpose(1, 2), x[:, nx:].reshape(rhs, cy - 1, cx).transpose(1, 2))


def _join(gx, gy):
    f = lambda g: g.transpose(1, 2).reshape(g.shape[0], -1)  # noqa: E731
    return torch.cat([f(gx), f(gy)], dim=1)


class _Green:
    """x -> A x for [rhs, n] vectors through even embeddings of 2 cx x 2 cy."""

    def __init__(self, cx, cy, h, k):
        self.cx, self.cy, self.h = cx, cy, h
        E, XX, YY = _generators(cx, cy, h, k)
        self.spectra = [self._embed(g) for g in (E, XX, YY)]

    def _embed(self, g):
        if g.numel() == 0:
            return None
        px, py = 2 * self.cx, 2 * self.cy
        e = torch.zeros(px, py, dtype=torch.complex128, device=g.device)
        r, c = g.shape
        e[:r, :c] = g
        e[px - r + 1:, :c] = g[1:, :].flip(0)
        e[:, py - c + 1:] = e[:, 1:c].flip(1)
        return torch.fft.fft2(e)

    def _conv(self, g, s):
        r, c = g.shape[1:]
        out = torch.fft.ifft2(torch.fft.fft2(g, s=(2 * self.cx, 2 * self.cy)) * s)
        return out[:, :r, :c]

    def __call__(self, x):
        gx, gy = _split(x, self.cx, self.cy)
        faces = torch.zeros(x.shape[0], self.cx, self.cy, dtype=x.dtype, device=x.device)
        faces[:, :-1, :] += gx / self.h
        faces[:, 1:, :] -= gx / self.h
        faces[:, :, :-1] += gy / self.h
        faces[:, :, 1:] -= gy / self.h
        f = self._conv(faces, self.spectra[0])
        ox = gx if self.spectra[1] is None else self._conv(gx, self.spectra[1])
        oy = gy if self.spectra[2] is None else self._conv(gy, self.spectra[2])
        return _join(ox - (f[:, :-1, :] - f[:, 1:, :]) / self.h, oy - (f[:, :, :-1] - f[:, :, 1:]) / self.h)


class _Circulant:
    """The inverted partwise circulant approximation on the face grid."""

    def __init__(self, cx, cy, h, k, kernel):
        self.cx, self.cy = cx, cy
        dev = _device()
        E, XX, YY = (self._fold(g, kernel) for g in _generators(cx, cy, h, k))
        sx = torch.exp(2j * math.pi * torch.arange(cx, device=dev, dtype=torch.float64) / cx)[:, None]
        sy = torch.exp(2j * math.pi * torch.arange(cy, device=dev, dtype=torch.float64) / cy)[None, :]
        u, v = 1 - sx, 1 - sy
        xx, yy = XX - u.abs() ** 2 / h**2 * E, YY - v.abs() ** 2 / h**2 * E
        xy, yx = -u * v.conj() / h**2 * E, -u.conj() * v / h**2 * E
        if cy == 1:
            self.blocks = (1 / xx, None, None, None)
        else:
            d = xx * yy - xy * yx
            self.blocks = (yy / d, -xy / d, -yx / d, xx / d)

    def _fold(self, g, kernel):
        out = torch.zeros(self.cx, self.cy, dtype=torch.complex128, device=g.device)

        def weights(n, offsets):
            o = offsets.abs().double()
            if kernel == "rChan":
                return torch.ones_like(o)
            if kernel == "tChan":
                return (n - o) / n
            return torch.where(2 * o < n, 1.0, torch.where(2 * o == n, 0.5, 0.0)).double()

        def offsets(n, rows):
            o = torch.cat([torch.arange(n), torch.arange(1 - n, 0)]).to(g.device)
            return o[o.abs() < rows]

        if g.numel() == 0:
            return out
        ox, oy = offsets(self.cx, g.shape[0]), offsets(self.cy, g.shape[1])
        part = g[ox.abs()][:, oy.abs()] * weights(self.cx, ox)[:, None] * weights(self.cy, oy)[None, :]
        out.index_put_(((ox % self.cx)[:, None].expand_as(part), (oy % self.cy)[None, :].expand_as(part)), part,
                       accumulate=True)
        return torch.fft.fft2(out)

    def __call__(self, x):
        gx, gy = _split(x, self.cx, self.cy)
        s = (self.cx, self.cy)
        fx = torch.fft.fft2(gx, s=s)
        if self.cy == 1:
            ox, oy = self.blocks[0] * fx, fx
        else:
            fy = torch.fft.fft2(gy, s=s)
            ox = self.blocks[0] * fx + self.blocks[1] * fy
            oy = self.blocks[2] * fx + self.blocks[3] * fy
        return _join(torch.fft.ifft2(ox)[:, :self.cx - 1, :], torch.fft.ifft2(oy)[:, :, :self.cy - 1])


class _BlockJacobi:
    """The inverses of the Green's matrix's diagonal blocks over 2 x 2 faces. A block's matrix depends on which
    of its rooftops exist alone, so there are four at most: inner, last column, last row, last corner."""

    def __init__(self, cx, cy, h, k):
        self.cx, self.cy = cx, cy
        E, XX, YY = (g.cpu() for g in _generators(cx, cy, h, k))
        nx = (cx - 1) * cy
        groups = {}
        for J in range(0, cy, 2):
            for I in range(0, cx, 2):
                roof = [(0, i, j) for j in range(J, min(J + 2, cy)) for i in range(I, min(I + 2, cx - 1))]
                roof += [(1, i, j) for j in range(J, min(J + 2, cy - 1)) for i in range(I, min(I + 2, cx))]
                shape = tuple((d, i - I, j - J) for d, i, j in roof)
                index = [i + (cx - 1) * j if d == 0 else nx + i + cx * j for d, i, j in roof]
                groups.setdefault(shape, []).append(index)

        def entry(p, q):
            z = (XX, YY)[p[0]][abs(p[1] - q[1]), abs(p[2] - q[2])] if p[0] == q[0] else 0
            for s in range(2):
                for t in range(2):
                    fx = (p[1] + s * (p[0] == 0)) - (q[1] + t * (q[0] == 0))
                    fy = (p[2] + s * (p[0] == 1)) - (q[2] + t * (q[0] == 1))
                    z = z - (1.0 if s == t else -1.0) / h**2 * E[abs(fx), abs(fy)]
            return z

        self.groups = []
        for shape, index in groups.items():
            if shape:
                m = torch.tensor([[complex(entry(p, q)) for q in shape] for p in shape], dtype=torch.complex128)
                self.groups.append((torch.tensor(index, device=_device()), torch.linalg.inv(m).to(_device())))

    def __call__(self, x):
        y = torch.empty_like(x)
        for index, inv in self.groups:
            y[:, index] = x[:, index] @ inv.T
        return y


def _exact_preconditioner(cx, cy, h, k, pc):
    if pc == "none":
        return None
    return _BlockJacobi(cx, cy, h, k) if pc == "blockJacobi" else _Circulant(cx, cy, h, k, pc)


def _exact_wave(cx, cy, h, k, direction, polarization):
    """The rooftops' integrals of a unit plane wave by the 8-point rule that assembly uses as well."""
    p, w = _rule(8)
    sx, sy = -1j * k * direction[0] * h, -1j * k * direction[1] * h
    one = lambda s: (torch.exp(s * p) * w).sum()  # noqa: E731
    hat = lambda s: (torch.exp(s * p) * w * (p + cmath.exp(s) * (1 - p))).sum()  # noqa: E731
    parts = []
    for pol, ref, rows, cols in ((polarization[0], hat(sx) * one(sy), cx - 1, cy),
                                 (polarization[1], one(sx) * hat(sy), cx, cy - 1)):
        ex = torch.exp(sx * torch.arange(rows, device=_device(), dtype=torch.float64))
        ey = torch.exp(sy * torch.arange(cols, device=_device(), dtype=torch.float64))
        parts.append((pol * h * h * ref * ey[:, None] * ex[None, :]).reshape(-1))
    return torch.cat(parts)


def _exact_cocg(A, M, b, iterations, tolerance=0.0):
    """[rhs, n]: the solutions and residual histories after the given iterations, or to a tolerance."""
    x, r = torch.zeros_like(b), b.clone()
    bn = torch.linalg.vector_norm(b, dim=1)
    history = [torch.ones_like(bn)]
    d = rho = None
    for _ in range(iterations):
        z = r if M is None else M(r)
        nxt = (r * z).sum(1)
        d = z.clone() if d is None else z + (nxt / rho)[:, None] * d
        rho = nxt
        q = A(d)
        alpha = rho / (d * q).sum(1)
        x = x + alpha[:, None] * d
        r = r - alpha[:, None] * q
        history.append(torch.linalg.vector_norm(r, dim=1) / bn)
        if float(history[-1].max()) < tolerance:
            break
    return x, torch.stack(history, dim=1)


def _exact_gmres(A, M, b, iterations, restart, side):
    """One right-hand side [1, n]: restarted GMRES, its least-squares problems solved from the Hessenberg."""
    P = M if side == "left" and M is not None else (lambda v: v)
    N = M if side == "right" and M is not None else (lambda v: v)
    x, r, done = torch.zeros_like(b), P(b), 0
    ref = torch.linalg.vector_norm(r)
    history = [1.0]
    while done < iterations:
        m = min(restart, iterations - done)
        rn = torch.linalg.vector_norm(r)
        V = torch.zeros(m + 1, b.shape[1], dtype=b.dtype, device=b.device)
        H = torch.zeros(m + 1, m, dtype=b.dtype, device=b.device)
        V[0] = r[0] / rn
        for j in range(m):
            w = P(A(N(V[j:j + 1])))[0]
            for _ in range(2):
                c = V[:j + 1].conj() @ w
                w = w - c @ V[:j + 1]
                H[:j + 1, j] += c
            H[j + 1, j] = torch.linalg.vector_norm(w)
            V[j + 1] = w / H[j + 1, j]
        Hc = H.cpu().numpy()
        y = None
        for j in range(m):
            g = np.zeros(j + 2, np.complex128)
            g[0] = float(rn)
            q, t = np.linalg.qr(Hc[:j + 2, :j + 1], mode="complete")
            qg = q.conj().T @ g
            history.append(float(abs(qg[-1])) / float(ref))
            if j == m - 1:
                y = np.linalg.solve(t[:j + 1], qg[:j + 1])
        x = x + N((torch.from_numpy(y).to(b.device) @ V[:m])[None])
        r = P(b - A(x))
        done += m
    return x, torch.tensor(history, dtype=torch.float64)


def _exact_solve(cx, cy, h, k, method, pc, side, b, iterations):
    A, M = _Green(cx, cy, h, k), _exact_preconditioner(cx, cy, h, k, pc)
    if method == "cg":
        return _exact_cocg(A, M, b, iterations)
    got = [_exact_gmres(A, M, row[None], iterations, 50, side) for row in b]
    return torch.cat([g[0] for g in got]), torch.stack([g[1] for g in got])


def exact(case, seed):
    kind, h = case["kind"], 1.0 / case["density"]
    k = _wavenumber(seed)
    if kind in ("product", "circulant"):
        cx, cy, n = case["cx"], case["cy"], _rooftops(case["cx"], case["cy"])
        x = _vector(seed, n * case["rhs"], case["precision"], _device()).to(torch.complex128).reshape(-1, n)
        op = _Green(cx, cy, h, k) if kind == "product" else _Circulant(cx, cy, h, k, case["kernel"])
        return op(x).reshape(-1)
    if kind == "setup":
        cx, cy = case["cx"], case["cy"]
        x = _vector(seed, _rooftops(cx, cy), "double", _device())[None]
        return {"product": _Green(cx, cy, h, k)(x)[0],
                "preconditioned": _exact_preconditioner(cx, cy, h, k, case["pc"])(x)[0],
                "wave": _exact_wave(cx, cy, h, k, *_waves(seed, 1)[0])}
    if kind == "solve":
        cx, cy = case["cx"], case["cy"]
        b = torch.stack([_exact_wave(cx, cy, h, k, d, p) for d, p in _waves(seed, case["rhs"])])
        x, history = _exact_solve(cx, cy, h, k, case["method"], case["pc"], case["side"], b, case["iterations"])
        if case["rhs"] > 1:
            return {"x": list(x), "history": list(history), "iterations": [case["iterations"]] * case["rhs"]}
        rcs = (k * Z0) ** 2 * float((b[0] * x[0]).sum().abs()) ** 2 / (4 * math.pi)
        return {"x": x[0], "history": history[0], "iterations": case["iterations"], "rcs": rcs}
    if kind == "strip":
        cx = case["cx"]
        b = torch.zeros(1, cx - 1, dtype=torch.complex128, device=_device())
        port = cx // 2 - 1
        b[0, port] = h
        x, history = _exact_cocg(_Green(cx, 1, h, k), _Circulant(cx, 1, h, k, "rChan"), b, 1000, tolerance=1e-6)
        z = 1.0 / (h * complex(x[0, port]))
        return {"x": x[0], "iterations": history.shape[1] - 1, "impedance": [z.real, z.imag]}
    xs, histories = [], []
    for (cx, cy), (d, p) in zip(_uneven_sizes(case), _waves(seed, case["plates"])):
        x, history = _exact_solve(cx, cy, h, k, "gmres", "blockJacobi", "right",
                                  _exact_wave(cx, cy, h, k, d, p)[None], case["iterations"])
        xs.append(x[0])
        histories.append(history[0])
    return {"x": xs, "history": histories, "iterations": [case["iterations"]] * case["plates"]}
