"""Plain FP64 pipeline at the edges of its per-direction tables: fewer
velocities than lanes, odd counts per direction, h in 3D (KInner > 0),
velocity components outside the solution directions, and 1D grids too long for
the tables (the exponential per velocity).  Tolerance as for the other short
FP64 runs: max(1e-12, 4 x the distance of two FP64 restatements)."""
import numpy as np
import pytest

from conftest import rel_err

pytestmark = pytest.mark.gpu

FIELDS = ("rho", "U", "T", "q")


def _case(name):
    from dugksfoam_gb300 import cases

    if name == "nv25":
        return cases.cavity2d(n=9, nxi=5)
    if name == "odd33":
        return cases.cavity2d(n=6, nxi=33)
    if name == "uz":
        c = cases.cavity2d(n=7, nxi=9)
        c["U0"][:, 2] = 5.0
        return c
    if name == "hexK2":
        c = cases.cavity3d(n=4, nxi=7)
        c["gas"] = dict(c["gas"], KInner=2)
        return c
    return cases.tube1d(nx=12, nxi=int(name[4:]))


@pytest.mark.parametrize("name", ["nv25", "odd33", "uz", "hexK2", "tube1900", "tube2900"])
def test_fp64_tables_match_oracle(built_lib, oracle_lib, name):
    from dugksfoam_gb300 import cases, solver
    from oracle.oracle import NumpyOracle, Oracle

    case, steps = _case(name), 8
    dt = cases.stable_dt(case)
    a, b = Oracle(case), NumpyOracle(case)
    a.step(dt, steps)
    b.step(dt, steps)
    want, other = a.cell(), b.cell()
    s = solver.FvDVM(case, precision=solver.FP64, pipeline=solver.PIPE_REFERENCE)
    s.set_dt(dt)
    s.evolution(steps)
    got = s.macros()
    s.close()
    for k in FIELDS:
        if not np.abs(want[k]).max() > 0:
            assert not np.abs(got[k]).max() > 0
            continue
        floor = rel_err(other[k], want[k])
        einf, el2 = rel_err(got[k], want[k])
        assert einf <= max(1e-12, 4 * floor[0]) and el2 <= max(1e-12, 4 * floor[1]), (name, k, einf, el2, floor)
