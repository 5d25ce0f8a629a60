"""Tangent-linear step on velocity grids whose tables fill the shared memory of
a block: with 351 and 352 velocities per direction a block of four entities
asks for the most that the moment kernel of the tangent leaves beside its own
totals.  adjoint . d = tangent(d) to 1e-9 of the sum of the terms' magnitudes
(the bound of the existing adjoint test); 353 takes two entities per block."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nxi", [350, 351, 352, 353])
def test_tangent_on_large_tables(built_lib, nxi):
    from dugksfoam_gb300 import cases, solver

    c = cases.cavity2d(n=3, nxi=nxi)
    rng = np.random.default_rng(1)
    c["Tb"] = c["Tb"] * (1 + 0.02 * rng.uniform(-1, 1, len(c["Tb"])))
    s = solver.FvDVM(c, precision=solver.FP64)
    s.set_dt(cases.case_dt(c))
    o = dict(n_steps=3, avg_first=1, q_patch=0, stress_patch=1, checkpoint_every=2)
    d = rng.standard_normal(s.info()["n_wall_faces"])
    J, g, gs = s.objective_adjoint(**o)
    Jt, dJ = s.objective_tangent(d, 0.7, **o)
    s.close()
    scale = np.abs(g * d).sum() + abs(0.7 * gs)
    assert scale > 0 and abs(J - Jt) <= 1e-10 * max(abs(J), abs(Jt))
    assert abs(g @ d + 0.7 * gs - dJ) <= 1e-9 * scale
