"""Components and iterations that have stopped cost no preconditioner applications:
device times of one solve against another of the same sizes, several times apart."""
import dataclasses

import numpy as np
import pytest

from rheotool_gb300 import abi
from rheotool_gb300.case import SolverControl, cavity_case
from rheotool_gb300.mesh import cavity_mesh, channel_mesh

from test_gpu_parity import laplacian_system

pytestmark = pytest.mark.gpu


def test_batched_momentum_solve_skips_stopped_components():
    """Cavities from rest: the y component starts converged, and the solve takes
    clearly less than one in which both iterate (0.68 of it; with a V-cycle for
    the stopped component, 1.1)."""
    from rheotool_gb300.batch import BatchContext
    mesh = cavity_mesh(96)
    ms = {}
    for kick in (0.0, 0.1):
        cases = [cavity_case(96, mesh=mesh) for _ in range(96)]
        for c in cases:
            c.precision = abi.RT_PREC_MIXED
        bt = BatchContext(cases)
        try:
            f = bt.ctx.fields()
            f.U[:, 1] = kick * np.random.default_rng(0).normal(size=bt.nCells)
            times = []
            for _ in range(3):
                bt.ctx.set_fields(f)
                bt.ctx.profile(True)
                bt.step(1)
                times.append(bt.ctx.profile_report()["batch_bicgstab_persistent"][1])
                bt.ctx.profile(False)
            iters = [bt.case_perf()[0].U[k].nIterations for k in range(2)]
        finally:
            bt.ctx.close()
        assert iters[0] > 5 and (iters[1] == 0 if kick == 0.0 else iters[1] > 5)
        ms[kick] = min(times)
    assert ms[0.0] < 0.85 * ms[0.1], ms


@pytest.mark.parametrize("precision", [abi.RT_PREC_FP64, abi.RT_PREC_MIXED])
def test_sweeps_launched_ahead_of_the_poll_return_at_once(ctx, precision):
    """PCG on a mesh without box structure launches sixteen iterations before the
    host can see that the first met the tolerance: the sweeps of the other
    fifteen together take less than a half of sixteen that iterate (a tenth)."""
    mesh = dataclasses.replace(channel_mesh(200, 190, 1), shape=None, cellIJK=None)
    rng = np.random.default_rng(1)
    system = laplacian_system(mesh, rng)
    b = rng.normal(size=(1, mesh.nCells)) * mesh.V
    ctx.upload_mesh(mesh)
    scope = "dilu_precondition" if precision == abi.RT_PREC_FP64 else "dilu_precondition32"
    ms = {}
    try:
        ctx.set_precision(precision)
        # (the mixed form's tolerance is two decades tighter)
        for n, tolerance, budget in ((16, 1e-300, 16), (1, 0.9 if precision == abi.RT_PREC_FP64 else 90.0, 1000)):
            times = []
            for _ in range(3):
                ctx.profile(True)
                p = ctx.ldu_solve(*system, b, np.zeros_like(b), SolverControl("PCG", "DIC", tolerance, 0.0, 0, budget))[0]
                launches, t, _ = ctx.profile_report()[scope]
                ctx.profile(False)
                assert launches == 16 and p.nIterations == n
                times.append(t)
            ms[n] = min(times)
    finally:
        ctx.set_precision(abi.RT_PREC_FP64)
    assert ms[1] < 0.5 * ms[16], ms
