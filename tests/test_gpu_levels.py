"""The level-scheduled DIC/DILU sweeps (one kernel an application) on meshes
without box structure: against the FP64 oracle's iterates, with levels of one
cell, levels wider than a CTA's threads, a mesh too large for its shared memory
(values in global memory) and one whose levels a cluster of CTAs walks."""
import dataclasses

import numpy as np
import pytest

from rheotool_gb300 import abi
from rheotool_gb300.case import SolverControl, contraction_case
from rheotool_gb300.mesh import channel_mesh, contraction_mesh

pytestmark = pytest.mark.gpu


MESHES = {
    "row": lambda: channel_mesh(40, 1, 1),                    # one cell a level
    "plane": lambda: contraction_mesh(30, 20, 20, 11, two_d=True),
    "block": lambda: channel_mesh(17, 13, 9),
    "global": lambda: channel_mesh(200, 190, 1),              # 38,000 cells: more than 220 KB in FP64
    "wide": lambda: channel_mesh(50, 44, 44),                 # levels of 1,900 cells: several passes
    "cluster": lambda: channel_mesh(66, 66, 66),              # levels of 3,270 cells: a cluster of eight
    "chain": lambda: channel_mesh(60000, 1, 1),               # more levels than shared memory holds starts of
}


def system(mesh, rng, asym):
    """A diagonally dominant LDU system (an upwinded convection-diffusion one with asym > 0)."""
    N = mesh.nCells
    g = mesh.magSf * mesh.deltaCoeffs * (1.0 + rng.random(mesh.nFaces))
    flux = asym * mesh.magSf * rng.normal(size=mesh.nFaces)
    upper, lower = -g + np.minimum(flux, 0.0), -g - np.maximum(flux, 0.0)
    diag = -(np.bincount(mesh.owner, upper, N) + np.bincount(mesh.neighbour, lower, N)) + 1e-2 * g.max()
    return diag, upper, lower


@pytest.mark.parametrize("solver,pre,asym,nc", [("PCG", "DIC", 0.0, 1), ("PBiCGStab", "DILU", 1.0, 3),
                                                ("PBiCG", "DILU", 1.0, 1)])
@pytest.mark.parametrize("name", sorted(MESHES))
def test_level_sweeps_match_the_oracle(ctx, name, solver, pre, asym, nc):
    from oracle.pyoracle import Oracle
    mesh = dataclasses.replace(MESHES[name](), shape=None, cellIJK=None)
    rng = np.random.default_rng(41)
    diag, upper, lower = system(mesh, rng, asym)
    b = rng.normal(size=(nc, mesh.nCells)) * mesh.V.mean()
    # six iterations: both sides evaluate the same recurrences, before BiCGStab
    # amplifies their reductions' different rounding
    ctl = SolverControl(solver, pre, 1e-30, 0.0, 0, 6)
    ctx.upload_mesh(mesh)
    x = np.zeros((nc, mesh.nCells))
    perf = ctx.ldu_solve(diag, upper, lower, b, x, ctl)
    orc = Oracle(contraction_case(mesh))
    for k in range(nc):
        xo = np.zeros(mesh.nCells)
        po = orc.ldu_solve(diag, upper, lower, b[k].copy(), xo, ctl)
        assert perf[k].nIterations == po.nIterations
        assert np.linalg.norm(x[k] - xo) <= 1e-9 * np.linalg.norm(xo)


@pytest.mark.parametrize("name", sorted(MESHES))
def test_level_sweeps_mixed_meet_the_fp64_residual(ctx, name):
    mesh = dataclasses.replace(MESHES[name](), shape=None, cellIJK=None)
    rng = np.random.default_rng(42)
    diag, upper, lower = system(mesh, rng, 1.0)
    b = rng.normal(size=(2, mesh.nCells)) * mesh.V.mean()
    ctx.upload_mesh(mesh)
    try:
        ctx.set_precision(abi.RT_PREC_MIXED)
        x = np.zeros((2, mesh.nCells))
        perf = ctx.ldu_solve(diag, upper, lower, b, x, SolverControl("PBiCGStab", "DILU", 1e-9, 0.0, 0, 200))
    finally:
        ctx.set_precision(abi.RT_PREC_FP64)
    for k in range(2):
        assert perf[k].converged
        assert ctx.residual(diag, upper, lower, b[k], x[k]) < 1e-9
