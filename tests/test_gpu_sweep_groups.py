"""The structured sweeps' groups of tiles: two tiles a CTA where such groups run
all at once, four where they do not, and what RT_OPT_SWEEP_TUNE forces; every
choice the same bits, and the schedule that rt_sweep_schedule reports the one that
ran."""
import numpy as np
import pytest

from rheotool_gb300 import abi
from rheotool_gb300.case import SolverControl
from rheotool_gb300.mesh import cavity_mesh, channel_mesh, contraction_mesh

from test_gpu_parity import laplacian_system

pytestmark = pytest.mark.gpu

MIXED_PRECOND_DEFAULT = MIXED_PRECOND_U_DEFAULT = -2
NARROW, WIDE = {"candidate": 2, "P": 16, "NB": 3}, {"candidate": 1, "P": 8, "NB": 5}


def solve(ctx, system, b, solver, precision, budget, tune=0, sweep=abi.SWEEP_SYSTOLIC):
    """psi and the iteration counts, with the exact sweeps."""
    pre = "DIC" if solver == "PCG" else "DILU"
    x = np.zeros_like(b)
    try:
        ctx.set_option(abi.RT_OPT_MIXED_PRECOND, 0)
        ctx.set_option(abi.RT_OPT_MIXED_PRECOND_U, 0)
        ctx.set_option(abi.RT_OPT_SWEEP_TUNE, tune)
        ctx.set_sweep(sweep)
        ctx.set_precision(precision)
        perf = ctx.ldu_solve(*system, b, x, SolverControl(solver, pre, 1e-13, 0.0, 0, budget))
        schedule = ctx.sweep_schedule()["fp64" if precision == abi.RT_PREC_FP64 else "fp32"]
    finally:
        ctx.set_precision(abi.RT_PREC_FP64)
        ctx.set_sweep(abi.SWEEP_AUTO)
        ctx.set_option(abi.RT_OPT_SWEEP_TUNE, 0)
        ctx.set_option(abi.RT_OPT_MIXED_PRECOND, MIXED_PRECOND_DEFAULT)
        ctx.set_option(abi.RT_OPT_MIXED_PRECOND_U, MIXED_PRECOND_U_DEFAULT)
    return x, [p.nIterations for p in perf], schedule


# rows (j, k) of ny x nz, tiles of 8 x 4: 100 x 100 is 7 x 25 groups of two tiles, more
# than the GPU's 152 SMs, and so are three components of 100 x 40
@pytest.mark.parametrize("precision", [abi.RT_PREC_FP64, abi.RT_PREC_MIXED])
@pytest.mark.parametrize("ny,nz,nc,want", [(100, 100, 1, WIDE), (100, 40, 1, NARROW), (100, 40, 3, WIDE), (30, 20, 3, NARROW)])
def test_reported_schedule_is_the_one_that_ran(ctx, precision, ny, nz, nc, want):
    mesh = channel_mesh(6, ny, nz)
    rng = np.random.default_rng(81)
    system = laplacian_system(mesh, rng, asym=0.0 if nc == 1 else 3.0)
    b = rng.normal(size=(nc, mesh.nCells)) * mesh.V
    ctx.upload_mesh(mesh)
    assert ctx.sweep_schedule()["fp64"]["candidate"] == -1 and ctx.sweep_schedule()["fp32"]["candidate"] == -1
    _, _, schedule = solve(ctx, system, b, "PCG" if nc == 1 else "PBiCGStab", precision, 2)
    assert schedule == want
    _, _, schedule = solve(ctx, system, b, "PCG" if nc == 1 else "PBiCGStab", precision, 2, tune=5)
    assert schedule == {"candidate": 4, "P": 4, "NB": 6}


SHAPES = {
    "groups past the SMs": lambda: channel_mesh(6, 100, 100),       # four tiles by default
    "one plane": lambda: cavity_mesh(21, 130),                      # tiles of 32 rows
    "holes": lambda: contraction_mesh(12, 10, 30, 10, 11, 4.0, 4.0),
    "odd edges": lambda: channel_mesh(17, 9, 5),                    # a row and a plane past the tiles
}


@pytest.mark.parametrize("nc", [1, 3, 6])
@pytest.mark.parametrize("name", sorted(SHAPES))
def test_every_group_shape_gives_the_same_bits(ctx, name, nc):
    """All schedules against the level-scheduled sweeps in FP64, and against each
    other in FP32 (whose sweeps take the i term before the j term, as the level
    sweeps do not)."""
    mesh = SHAPES[name]()
    rng = np.random.default_rng(82)
    system = laplacian_system(mesh, rng, asym=3.0)
    b = rng.normal(size=(nc, mesh.nCells)) * mesh.V
    ctx.upload_mesh(mesh)
    want, iters, _ = solve(ctx, system, b, "PBiCGStab", abi.RT_PREC_FP64, 6, sweep=abi.SWEEP_LEVELS)
    want32 = None
    for tune in range(6):
        x, n, _ = solve(ctx, system, b, "PBiCGStab", abi.RT_PREC_FP64, 6, tune)
        assert n == iters and np.array_equal(x, want), tune
        x, n32, _ = solve(ctx, system, b, "PBiCGStab", abi.RT_PREC_MIXED, 6, tune)
        if want32 is None:
            want32, iters32 = x, n32
        assert n32 == iters32 and np.array_equal(x, want32), tune


@pytest.mark.parametrize("precision", [abi.RT_PREC_FP64, abi.RT_PREC_MIXED])
def test_components_side_by_side_equal_one_by_one(ctx, precision):
    """Three components in one launch (four tiles a CTA on 100 x 40 rows) and each
    alone (two): the same bits."""
    mesh = channel_mesh(6, 100, 40)
    rng = np.random.default_rng(83)
    system = laplacian_system(mesh, rng, asym=3.0)
    b = rng.normal(size=(3, mesh.nCells)) * mesh.V
    ctx.upload_mesh(mesh)
    x, n, schedule = solve(ctx, system, b, "PBiCGStab", precision, 20)
    assert schedule == WIDE
    for k in range(3):
        xk, nk, schedule = solve(ctx, system, b[k:k + 1].copy(), "PBiCGStab", precision, 20)
        assert schedule == NARROW
        assert nk[0] == n[k] and np.array_equal(xk[0], x[k])
