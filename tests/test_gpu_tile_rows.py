"""FP32 face sweep with tiles whose cells do not divide among the block's 16
warps: the warps with a cell less relax more of the tile's rows.  Tile sizes
either side of multiples of 16, tiles smaller than the block, one cell per
tile; FP32 within 1e-5 of the oracle as the other short runs."""
import pytest

from conftest import rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("cells", [1, 5, 15, 16, 17, 24, 31, 33])
def test_tiles_match_oracle(built_lib, oracle_lib, monkeypatch, dim, cells):
    from dugksfoam_gb300 import cases, solver
    from oracle.oracle import Oracle

    monkeypatch.setenv("DUGKS_TILE_CELLS", str(cells))
    case, steps = cases.cavity2d(n=11, nxi=18) if dim == 2 else cases.cavity3d(n=5, nxi=8), 8
    dt = cases.stable_dt(case)
    ref = Oracle(case)
    ref.step(dt, steps)
    s = solver.FvDVM(case, precision=solver.FP32_FP64MOM)
    s.set_dt(dt)
    s.evolution(steps)
    got, want = s.macros(), ref.cell()
    s.close()
    for k in ("rho", "U", "T", "q"):
        assert rel_err(got[k], want[k])[0] <= 1e-5, (dim, cells, k)
