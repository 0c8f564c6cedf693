"""The mixed form's solver and preconditioner pairs beside PCG with DIC and PBiCGStab
with DILU: the options of the pressure solve's preconditioner (RT_OPT_MIXED_PRECOND)
are PCG's and those of the momentum solve's PBiCGStab's, so the other pairs make and
apply the factorisation of their matrix whatever the options say."""
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


@pytest.mark.parametrize("sweep", [abi.SWEEP_AUTO, abi.SWEEP_LEVELS])
@pytest.mark.parametrize("option,option_u,nc", [(-2, -2, 1), (-2, -2, 3), (4, -2, 1), (4, 0, 1), (0, -2, 2), (-1, -2, 1)])
def test_mixed_pcg_with_dilu_applies_what_it_prepared(option, option_u, nc, sweep):
    """PCG with DILU in the mixed form: RT_OPT_MIXED_PRECOND_U is PBiCGStab's, so the
    factorisation, or its Jacobi sweeps, of this matrix are made and applied."""
    from rheotool_gb300.runtime import Context
    mesh = contraction_mesh(12, 10, 30, 10, 6, 4.0, 4.0)
    rng = np.random.default_rng(64)
    system = laplacian_system(mesh, rng, shift=30.0)
    b = rng.normal(size=(nc, mesh.nCells)) * mesh.V
    ctl = SolverControl("PCG", "DILU", 1e-10, 0.0, 0, 500)
    with Context(0) as c:     # (a context with no earlier factorisation)
        c.upload_mesh(mesh)
        c.set_sweep(sweep)
        c.set_precision(abi.RT_PREC_MIXED)
        c.set_option(abi.RT_OPT_MIXED_PRECOND, option)
        c.set_option(abi.RT_OPT_MIXED_PRECOND_U, option_u)
        x = np.zeros_like(b)
        perf = c.ldu_solve(*system, b, x, ctl)
        for k in range(nc):
            assert perf[k].converged and c.residual(*system, b[k], x[k]) < 1e-10
    with Context(0) as c:
        c.upload_mesh(mesh)
        x64 = np.zeros_like(b)
        p64 = c.ldu_solve(*system, b, x64, ctl)
    # (two decades tighter in the mixed form, and Jacobi sweeps in place of exact ones)
    assert all(perf[k].nIterations <= 4 * p64[k].nIterations + 20 for k in range(nc))
