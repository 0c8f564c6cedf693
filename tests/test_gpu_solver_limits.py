"""Solver controls at their limits: an iteration budget of zero, which every
solver of OpenFOAM's do-while loops (PBiCGStab.C's do { ... } while) spends one
iteration on when it starts unconverged."""
import dataclasses

import numpy as np
import pytest

from rheotool_gb300 import abi
from rheotool_gb300.case import SolverControl, contraction_case
from rheotool_gb300.mesh import contraction_mesh

from test_gpu_parity import laplacian_system, rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("structured", [True, False])
@pytest.mark.parametrize("precision", [abi.RT_PREC_FP64, abi.RT_PREC_MIXED])
def test_pbicgstab_without_a_budget_makes_one_iteration(ctx, structured, precision):
    """maxIter 0: a component that starts converged takes none, the others one,
    with the psi of maxIter 1; in FP64 the oracle's."""
    from oracle.pyoracle import Oracle
    mesh = contraction_mesh(12, 10, 30, 10, 6, 4.0, 4.0)
    if not structured:
        mesh = dataclasses.replace(mesh, shape=None, cellIJK=None)
    rng = np.random.default_rng(61)
    diag, upper, lower = laplacian_system(mesh, rng, asym=3.0)
    b = rng.normal(size=(3, mesh.nCells)) * mesh.V
    b[1] = 0.0
    ctx.upload_mesh(mesh)
    out = {}
    try:
        ctx.set_precision(precision)
        for budget in (0, 1):
            x = np.zeros_like(b)
            ctl = SolverControl("PBiCGStab", "DILU", 1e-12, 0.0, 0, budget)
            perf = ctx.ldu_solve(diag, upper, lower, b, x, ctl)
            out[budget] = (x, [p.nIterations for p in perf], [p.finalResidual for p in perf])
    finally:
        ctx.set_precision(abi.RT_PREC_FP64)
    assert out[0][1] == [1, 0, 1] and out[0][1:] == out[1][1:]
    assert np.array_equal(out[0][0], out[1][0])
    if precision == abi.RT_PREC_FP64:
        orc = Oracle(contraction_case(mesh))
        for k in range(3):
            xo = np.zeros(mesh.nCells)
            po = orc.ldu_solve(diag, upper, lower, b[k].copy(), xo, SolverControl("PBiCGStab", "DILU", 1e-12, 0.0, 0, 0))
            assert po.nIterations == out[0][1][k]
            assert rel(out[0][0][k], xo) < 1e-9


@pytest.mark.parametrize("structured", [True, False])
@pytest.mark.parametrize("precision", [abi.RT_PREC_FP64, abi.RT_PREC_MIXED])
def test_pcg_without_a_budget_makes_one_iteration(ctx, structured, precision):
    """The same of PCG, whose batched form makes one too."""
    from oracle.pyoracle import Oracle
    mesh = contraction_mesh(12, 10, 30, 10, 6, 4.0, 4.0)
    if not structured:
        mesh = dataclasses.replace(mesh, shape=None, cellIJK=None)
    rng = np.random.default_rng(63)
    system = laplacian_system(mesh, rng)
    b = rng.normal(size=(1, mesh.nCells)) * mesh.V
    ctx.upload_mesh(mesh)
    out = {}
    try:
        ctx.set_precision(precision)
        for budget in (0, 1):
            x = np.zeros_like(b)
            perf = ctx.ldu_solve(*system, b, x, SolverControl("PCG", "DIC", 1e-12, 0.0, 0, budget))[0]
            out[budget] = (x, perf.nIterations, perf.finalResidual)
    finally:
        ctx.set_precision(abi.RT_PREC_FP64)
    assert out[0][1] == 1 and out[0][1:] == out[1][1:]
    assert np.array_equal(out[0][0], out[1][0])
    if precision == abi.RT_PREC_FP64:
        xo = np.zeros(mesh.nCells)
        po = Oracle(contraction_case(mesh)).ldu_solve(*system, b[0].copy(), xo, SolverControl("PCG", "DIC", 1e-12, 0.0, 0, 0))
        assert po.nIterations == 1 and rel(out[0][0][0], xo) < 1e-9


@pytest.mark.parametrize("precision", [abi.RT_PREC_FP64, abi.RT_PREC_MIXED])
@pytest.mark.parametrize("budget", [-2, -5])
def test_batch_below_zero_budget_makes_one_iteration(precision, budget):
    """A small batch (the launch path) with a negative maxIter: the step of maxIter 0."""
    from rheotool_gb300.batch import BatchContext, cavity_sweep
    out = {}
    for n in (0, budget):
        cases = cavity_sweep(n_cases=3, n_min=8, n_max=20, seed=7, dt=5e-3, precision=precision)
        for c in cases:
            for s in (c.solverP, c.solverU, c.solverTheta):
                s.maxIter = n
        bt = BatchContext(cases)
        try:
            bt.step(1)
            f = bt.ctx.fields()
            out[n] = ([(p.p.nIterations, p.U[0].nIterations, p.theta[0].nIterations) for p in bt.case_perf()], f)
        finally:
            bt.ctx.close()
    assert out[budget][0] == out[0][0] == [(1, 1, 1)] * 3
    for name in ("U", "p", "theta"):
        assert np.array_equal(getattr(out[budget][1], name), getattr(out[0][1], name)), name
