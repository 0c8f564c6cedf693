"""Components and iterations that have stopped cost no preconditioner applications:
device times of one solve against another of the same sizes, several times apart."""
import numpy as np
import pytest

from rheotool_gb300 import abi
from rheotool_gb300.case import cavity_case
from rheotool_gb300.mesh import cavity_mesh

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
