"""FP32 cell gather: the order in which the warps take the cells, at meshes of
less than one, one to two and up to four cells per warp (2,432 warps on 152
SMs), where cells with boundary faces are moved to warps without a cell in the
last round, and where too many of them are left.  Every cell is taken once: all
fields within 1e-5 of the oracle as the other short runs."""
import pytest

from conftest import rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,n", [(2, 49), (2, 50), (2, 66), (2, 69), (2, 72), (2, 90), (3, 14), (3, 17)])
def test_every_cell_is_gathered_once(built_lib, oracle_lib, dim, n):
    from dugksfoam_gb300 import cases, solver
    from oracle.oracle import Oracle

    case, steps = (cases.cavity2d(n=n, nxi=8) if dim == 2 else cases.cavity3d(n=n, nxi=4)), 4
    dt = cases.stable_dt(case)
    ref = Oracle(case)
    ref.step(dt, steps)
    s = solver.FvDVM(case, precision=solver.FP32_FP64MOM)
    s.set_dt(dt)
    s.evolution(steps)
    got, want = s.macros(), ref.cell()
    s.close()
    for k in ("rho", "U", "T", "q"):
        assert rel_err(got[k], want[k])[0] <= 1e-5, (dim, n, k)
