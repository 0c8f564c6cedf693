"""The mixed PBiCGStab with DIC on one component: the options of the mixed pressure
solve's preconditioner (RT_OPT_MIXED_PRECOND) are PCG's, so it takes the exact
FP32 sweeps whatever they say."""
import numpy as np
import pytest

from rheotool_gb300 import abi
from rheotool_gb300.case import SolverControl
from rheotool_gb300.mesh import contraction_mesh

from test_gpu_parity import laplacian_system

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("option", [-2, -1, 0, 4])
def test_mixed_pbicgstab_with_dic_uses_this_matrix_sweeps(option):
    from rheotool_gb300.runtime import Context
    mesh = contraction_mesh(12, 10, 30, 10, 6, 4.0, 4.0)
    rng = np.random.default_rng(62)
    system = laplacian_system(mesh, rng, shift=30.0)
    b = rng.normal(size=(1, mesh.nCells)) * mesh.V
    ctl = SolverControl("PBiCGStab", "DIC", 1e-10, 0.0, 0, 500)
    with Context(0) as c:     # (a context with no earlier factorisation)
        c.upload_mesh(mesh)
        x64 = np.zeros_like(b)
        p64 = c.ldu_solve(*system, b, x64, ctl)[0]
    with Context(0) as c:
        c.upload_mesh(mesh)
        c.set_precision(abi.RT_PREC_MIXED)
        c.set_option(abi.RT_OPT_MIXED_PRECOND, option)
        x = np.zeros_like(b)
        p = c.ldu_solve(*system, b, x, ctl)[0]
        assert p.converged and c.residual(*system, b, x) < 1e-10
    # (two decades tighter in the mixed form)
    assert p.nIterations <= 2 * p64.nIterations + 20
