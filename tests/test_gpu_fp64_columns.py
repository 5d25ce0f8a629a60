"""Plain FP64 pipeline where lanes own columns of velocities along the last
direction: either side of the share of busy lanes from which columns are taken
(2D 23 | 24 velocities per direction for the moments, 28 | 29 for the
relaxation; 3D 6 | 7), one and two rounds of columns, remainders of the batches
of four, more velocities than a wall thread has sign bits for (17^3), h in 3D,
flows and walls that move in every direction (moments about the old velocity,
wall stress and heat flux of the same sums).  Tolerance of cells as for the
other short FP64 runs: max(1e-12, 4 x the distance of two FP64 restatements); of
walls as in the parity test of the small cases."""
import numpy as np
import pytest

from conftest import rel_err

pytestmark = pytest.mark.gpu

FIELDS = ("rho", "U", "T", "q")


def _case(name):
    from dugksfoam_gb300 import cases

    dim, nxi = name.split("-")[:2]
    if dim == "2d":
        c = cases.cavity2d(n=7, nxi=int(nxi), Tw=dict(fixedWalls=300.0))
    else:
        c = cases.cavity3d(n=4, nxi=int(nxi))
    if "K2" in name:
        c["gas"] = dict(c["gas"], KInner=2)
    D = 2 if dim == "2d" else 3
    rng = np.random.default_rng(7)
    fast = 1.2 if "fast" in name else 0.2  # in units of sqrt(2 R T)
    c0 = np.sqrt(2 * c["gas"]["R"] * 273.0)
    c["U0"][:, :D] = fast * c0 * np.array([0.7, -0.5, 0.4])[:D] + 5.0 * rng.standard_normal((len(c["U0"]), D))
    if "walls" in name:
        c["Ub"][:] = [20.0, -10.0, 30.0]
    return c


@pytest.mark.parametrize("name", ["2d-23", "2d-24", "2d-28", "2d-29", "2d-32", "2d-48", "2d-29-walls", "2d-28-fast",
                                  "3d-6", "3d-7", "3d-8", "3d-7-K2", "3d-9-walls",
                                  "3d-17-walls"])
def test_fp64_columns_match_oracle(built_lib, oracle_lib, name):
    from dugksfoam_gb300 import cases, solver
    from oracle.oracle import NumpyOracle, Oracle

    case, steps = _case(name), 4
    dt = cases.stable_dt(case)
    a, b = Oracle(case), NumpyOracle(case)
    a.step(dt, steps)
    b.step(dt, steps)
    want, other = a.cell(), b.cell()
    s = solver.FvDVM(case, precision=solver.FP64, pipeline=solver.PIPE_REFERENCE)
    s.set_dt(dt)
    s.evolution(steps)
    got = s.macros()
    for k in FIELDS:
        floor = rel_err(other[k], want[k])
        einf, el2 = rel_err(got[k], want[k])
        assert einf <= max(1e-12, 4 * floor[0]) and el2 <= max(1e-12, 4 * floor[1]), (name, k, einf, el2, floor)
    ow, nI = a.wall(), len(case["mesh"]["neighbour"])
    for pi, p in enumerate(case["mesh"]["patches"]):
        if p["type"] != "wall":
            continue
        w, sl = s.wall(pi, p["nFaces"]), slice(p["startFace"] - nI, p["startFace"] - nI + p["nFaces"])
        for k, tol in (("rhoW", 1e-12), ("qWall", 1e-11), ("stressWall", 1e-12)):
            assert rel_err(w[k], ow[k][sl])[0] <= tol, (name, p["name"], k)
    s.close()
