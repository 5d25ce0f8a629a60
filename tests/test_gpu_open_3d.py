"""FP32 open boundaries in 3D on a sheared box (oblique faces), on velocity
grids of whole and of split lane rows: within 1e-5 of the FP64 oracle (the FP32
path's bound)."""
import numpy as np
import pytest

from conftest import rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nxi", [8, 9, 12])
def test_fp32_open_faces_3d_match_oracle(built_lib, oracle_lib, nxi):
    from dugksfoam_gb300 import cases, solver
    from oracle.oracle import Oracle

    gas, rho0 = cases.gas_from_kn(0.1)
    mesh = cases.structured_mesh(5, 4, 4, two_d=False, patch_defs=[
        ("farfield", "patch", ["x0"], "farField"), ("outflow", "patch", ["x1"], "zeroGradient"),
        ("top", "patch", ["y1"], "fixedValue"), ("walls", "wall", ["y0", "z0", "z1"], None)])
    mesh["points"] = mesh["points"] @ np.array([[1.0, 0.0, 0.0], [0.37, 1.0, 0.0], [0.21, 0.29, 1.0]])
    case = cases.make_case(mesh, gas, rho0, nxi, 4.0 * np.sqrt(2 * gas["R"] * 273.0), two_d=False, lid_u=0.0, bvals={
        "farfield": dict(rho=rho0, T=300.0), "top": dict(rho=1.1 * rho0, U=(60.0, 0.0, 20.0), T=290.0),
        "outflow": dict(T=273.0)})
    dt = cases.cell_stable_dt(case)
    ref = Oracle(case)
    ref.step(dt, 6)
    s = solver.FvDVM(case, precision=solver.FP32_FP64MOM)
    s.set_dt(dt)
    s.evolution(6)
    got, want = s.macros(), ref.cell()
    s.close()
    for k in ("rho", "U", "T", "q"):
        einf, el2 = rel_err(got[k], want[k])
        assert einf <= 1e-5 and el2 <= 1e-5, (nxi, k, einf, el2)
