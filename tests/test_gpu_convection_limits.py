"""GaussDefCmpw's deferred correction where a gradient is not finite: the flux is
no number on every face of such a cell, also where the cell is downwind."""
import pytest

from rheotool_gb300 import abi
from rheotool_gb300.case import contraction_case
from rheotool_gb300.mesh import contraction_mesh

pytestmark = pytest.mark.gpu


def test_infinite_gradient_downwind_is_seen_at_once(ctx):
    """theta at the inlet face of the first cell so large that the cell's gradient
    overflows; the cell is downwind of all its faces and the inlet face carries no
    flux, so no other term holds the value."""
    from rheotool_gb300.runtime import RheoGpuError
    case = contraction_case(contraction_mesh(60, 10, 30, 10, 6, 4.0, 4.0))
    m = case.mesh
    ctx.setup_case(case)
    f = ctx.fields()
    inlet = m.patch("inlet")
    face = next(b for b in range(inlet.start, inlet.start + inlet.size) if m.bCell[b] == 0)
    f.phi[m.owner == 0] = -1e-6       # (cell 0 is the owner of all its internal faces)
    f.phib[:] = 0.0
    assert m.bmagSf[face] / m.V[0] > 4.0   # (times 1e308: infinite)
    f.thetab[face] = 1e308
    ctx.set_fields(f)
    with pytest.raises(RheoGpuError) as e:
        ctx.constitutive_correct()
    assert e.value.status == abi.RT_ENAN
