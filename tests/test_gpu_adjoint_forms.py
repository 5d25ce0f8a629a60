"""Adjoint against the tangent-linear step (the same FP64 step differentiated
the other way) over the forms the reverse passes are instantiated for: 2D with
odd velocity counts and ties, triangles, 3D with and without h, cells with more
faces than a warp stages, and more velocities per direction than the shared
memory of a default launch holds tables for.  adjoint . d = tangent(d) to 1e-9
of the sum of the terms' magnitudes (the bound of the existing adjoint test)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _case(name):
    from dugksfoam_gb300 import cases
    from test_gpu_polyhedra import merged

    gas, rho0 = cases.gas_from_kn(0.1)
    xi_max = 4.0 * np.sqrt(2 * gas["R"] * 273.0)
    if name == "quad9":
        return cases.cavity2d(n=6, nxi=9)
    if name == "tri8":
        return dict(cases.make_case(cases.delaunay_mesh(40, 5, seed=3), gas, rho0, 8, xi_max), unstructured=True)
    if name == "merged12":
        return cases.make_case(merged(cases.structured_mesh(12, 5, 1, two_d=True), 12, 5), gas, rho0, 12, xi_max)
    if name == "quad260":
        return cases.cavity2d(n=3, nxi=260)
    c = cases.cavity3d(n=3, nxi=7)
    if name == "hexK2":
        c["gas"] = dict(c["gas"], KInner=2)
    return c


@pytest.mark.parametrize("name", ["quad9", "tri8", "merged12", "quad260", "hex7", "hexK2"])
def test_adjoint_matches_tangent(built_lib, name):
    from dugksfoam_gb300 import cases, solver

    c = _case(name)
    rng = np.random.default_rng(0)
    c["Tb"] = c["Tb"] * (1 + 0.02 * rng.uniform(-1, 1, len(c["Tb"])))
    s = solver.FvDVM(c, precision=solver.FP64)
    s.set_dt(cases.case_dt(c))
    o = dict(n_steps=7, avg_first=3, q_patch=0, stress_patch=1, checkpoint_every=3)
    d = rng.standard_normal(s.info()["n_wall_faces"])
    J, g, gs = s.objective_adjoint(**o)
    Jt, dJ = s.objective_tangent(d, 0.7, **o)
    s.close()
    scale = np.abs(g * d).sum() + abs(0.7 * gs)
    assert scale > 0 and abs(J - Jt) <= 1e-10 * max(abs(J), abs(Jt))
    assert abs(g @ d + 0.7 * gs - dJ) <= 1e-9 * scale, (name, g @ d + 0.7 * gs, dJ)
