"""FP32 step with flows as fast as the thermal speed and twice that (the face
and cell moments are summed about velocity 0), lane rows of the velocity grid
whole and split, 2D and 3D: within 1e-5 of the FP64 oracle (the FP32 path's
bound)."""
import numpy as np
import pytest

from conftest import rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("speed", [1.0, 2.0])  # in units of sqrt(2 R T)
@pytest.mark.parametrize("dim, nxi", [("2d", 28), ("2d", 29), ("3d", 12), ("3d", 13)])
def test_fp32_fast_flow_matches_oracle(built_lib, oracle_lib, dim, nxi, speed):
    from dugksfoam_gb300 import cases, solver
    from oracle.oracle import Oracle

    case = cases.cavity2d(n=16, nxi=nxi) if dim == "2d" else cases.cavity3d(n=6, nxi=nxi)
    D = 2 if dim == "2d" else 3
    u = np.array([0.7, -0.6, 0.39])[:D]
    rng = np.random.default_rng(7)
    case["U0"][:, :D] = speed * np.sqrt(2 * case["gas"]["R"] * 273.0) * u / np.linalg.norm(u)
    case["U0"][:, :D] += 5.0 * rng.standard_normal((len(case["U0"]), D))
    dt = cases.stable_dt(case)
    ref = Oracle(case)
    ref.step(dt, 6)
    s = solver.FvDVM(case, precision=solver.FP32_FP64MOM)
    s.set_dt(dt)
    s.evolution(6)
    got, want = s.macros(), ref.cell()
    s.close()
    for k in ("rho", "U", "T", "q"):
        einf, el2 = rel_err(got[k], want[k])
        assert einf <= 1e-5 and el2 <= 1e-5, (k, einf, el2)
