"""The single-case V-cycle (mixed pressure and momentum solves) on matrices and
boxes at its edges: a diagonal that is zero in FP32, and boxes of one level."""
import numpy as np
import pytest

from rheotool_gb300 import abi
from rheotool_gb300.case import SolverControl
from rheotool_gb300.mesh import cavity_mesh, channel_mesh

pytestmark = pytest.mark.gpu


def solve(ctx, *args):
    try:
        ctx.set_precision(abi.RT_PREC_MIXED)
        return ctx.ldu_solve(*args)
    finally:
        ctx.set_precision(abi.RT_PREC_FP64)


def system(mesh, rng, asym):
    N = mesh.nCells
    g = mesh.magSf * mesh.deltaCoeffs * (1.0 + rng.random(mesh.nFaces))
    flux = asym * g * rng.normal(size=mesh.nFaces)
    up, lo = -g + np.minimum(flux, 0.0), -g - np.maximum(flux, 0.0)
    off = np.bincount(mesh.owner, up, N) + np.bincount(mesh.neighbour, lo, N)
    return -off + 1e-3 * np.abs(off).max(), up, lo


def detached(mesh, cell, diag, up, lo):
    """The system with one cell cut off, its diagonal 1e-60: zero in FP32."""
    diag, up, lo = diag.copy(), up.copy(), lo.copy()
    f = (mesh.owner == cell) | (mesh.neighbour == cell)
    np.add.at(diag, mesh.owner[f], up[f])       # (the diagonal is minus the couplings, and a shift)
    np.add.at(diag, mesh.neighbour[f], lo[f])
    up[f] = lo[f] = 0.0
    diag[cell] = 1e-60
    return diag, up, lo


CELLS = {"red": (8, 12), "black": (8, 13)}   # (i, j): i + j even, odd


@pytest.mark.parametrize("solver,pre,asym,nc", [("PCG", "DIC", 0.0, 1), ("PBiCGStab", "DILU", 0.3, 2)])
@pytest.mark.parametrize("colour", ["red", "black"])
def test_zero_diagonal_in_fp32_leaves_the_cell_alone(ctx, colour, solver, pre, asym, nc):
    """A cell that the V-cycle cannot divide by keeps its psi, also where an
    earlier matrix of the same mesh moved it; the other cells get their solution."""
    nx, ny = 41, 33
    mesh = cavity_mesh(nx, ny)
    i, j = CELLS[colour]
    cell = j * nx + i
    rng = np.random.default_rng(71)
    whole = system(mesh, rng, asym)
    cut = detached(mesh, cell, *whole)
    b = rng.normal(size=(nc, mesh.nCells))
    b[:, cell] = 0.0
    ctl = SolverControl(solver, pre, 1e-12, 0.0, 0, 500)
    ctx.upload_mesh(mesh)
    perf = solve(ctx, *whole, rng.normal(size=b.shape), np.zeros_like(b), ctl)
    assert all(p.converged for p in perf)
    x, x64 = np.zeros_like(b), np.zeros_like(b)
    x[:, cell] = x64[:, cell] = 0.75
    perf = solve(ctx, *cut, b, x, ctl)
    assert all(p.converged for p in perf)
    assert np.all(x[:, cell] == 0.75)
    ctx.ldu_solve(*cut, b, x64, ctl)
    x64[:, cell] = 0.75
    # (condition number below 1e4, residuals below 1e-12: see the box test of the V-cycle)
    assert np.linalg.norm(x - x64) <= 1e-8 * np.linalg.norm(x64)


def one_level_pcg(mesh, diag, up, b, tol, budget):
    """Iterations of flexible PCG with a one-level cycle in FP32: from x = 0 a red
    half-sweep, then sixteen times black and red, which is symmetric."""
    N = mesh.nCells
    o, n = mesh.owner, mesh.neighbour
    red = mesh.cellIJK.sum(axis=1) % 2 == 0
    up32, d32 = up.astype(np.float32), diag.astype(np.float32)

    def neighbours(x):
        y = np.zeros(N, np.float32)
        np.add.at(y, o, up32 * x[n])
        np.add.at(y, n, up32 * x[o])
        return y

    def cycle(r):
        r32, x = r.astype(np.float32), np.zeros(N, np.float32)
        for colour in [red] + [~red, red] * 16:
            x = np.where(colour, (r32 - neighbours(x)) / d32, x)
        return x.astype(np.float64)

    def amul(x):
        y = diag * x
        np.add.at(y, o, up * x[n])
        np.add.at(y, n, up * x[o])
        return y

    nf = np.abs(b).sum() + 1e-20   # (psi starts from zero)
    r, p, q, rho, alpha = b.copy(), None, None, 0.0, 0.0
    for it in range(1, budget + 1):
        w = cycle(r)
        beta = 0.0 if p is None else -alpha * (w @ q) / rho
        rho = w @ r
        p = w if p is None else w + beta * p
        q = amul(p)
        alpha = rho / (p @ q)
        r = r - alpha * q
        if np.abs(r).sum() / nf < tol:
            return it
    return budget


@pytest.mark.parametrize("dims", [(16, 16, 1), (22, 22, 1), (8, 8, 8), (128, 4, 1)])
def test_one_level_cycle_is_symmetric(ctx, dims):
    """A box of at most 512 cells is one level.  PCG needs a symmetric cycle: the
    library takes no more iterations than the reference loop with such a cycle
    (and two, for other roundings), on a Laplacian with one reference cell."""
    nx, ny, nz = dims
    mesh = cavity_mesh(nx, ny) if nz == 1 else channel_mesh(nx, ny, nz)
    rng = np.random.default_rng(72)
    N = mesh.nCells
    up = -mesh.magSf * mesh.deltaCoeffs * (1.0 + rng.random(mesh.nFaces))
    diag = -(np.bincount(mesh.owner, up, N) + np.bincount(mesh.neighbour, up, N))
    diag[0] *= 2.0
    b = rng.normal(size=N)
    tol = 1e-8
    want = one_level_pcg(mesh, diag, up, b, tol, 300)
    ctx.upload_mesh(mesh)
    try:
        ctx.set_option(abi.RT_OPT_MIXED_TIGHTEN, 0)
        x = np.zeros((1, N))
        perf = solve(ctx, diag, up, up, b, x, SolverControl("PCG", "DIC", tol, 0.0, 0, 300))[0]
    finally:
        ctx.set_option(abi.RT_OPT_MIXED_TIGHTEN, 2)
    assert perf.converged and want < 300
    assert perf.nIterations <= want + 2, (perf.nIterations, want)
