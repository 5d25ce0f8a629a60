"""Cells with more faces than the structured meshes have, and velocity counts
that are no multiples of the lane width: runs of 2 or 3 cells of a structured
mesh merged into one (6 and 8 faces in 2D, 10 and 14 in 3D, so that the face
groups of a warp, the staged face lists and their overflow are all used).
FP32 within 1e-5 of the oracle, FP64 within max(1e-12, 4 x the distance of two
FP64 restatements), as the other short runs."""
import numpy as np
import pytest

from conftest import rel_err

pytestmark = pytest.mark.gpu

FIELDS = ("rho", "U", "T", "q")


def merged(mesh, nx, run):
    """The mesh with every other group of `run` consecutive cells of a row merged into one cell."""
    nC, nI = mesh["n_cells"], len(mesh["neighbour"])
    i, row = np.arange(nC) % nx, np.arange(nC) // nx
    first = np.where((i // run + row) % 2 == 0, i // run * run, i)
    new = np.unique(row * nx + first, return_inverse=True)[1]
    own, nei = new[mesh["owner"]], new[mesh["neighbour"]]
    off, fv = mesh["face_offsets"], mesh["face_verts"]
    faces = [fv[off[f]:off[f + 1]] for f in range(len(off) - 1)]
    keep = np.nonzero(own[:nI] != nei)[0]
    keep = keep[np.lexsort((nei[keep], own[keep]))]
    assert (own[keep] < nei[keep]).all()
    order = np.concatenate([keep, np.arange(nI, len(faces))])
    out = dict(mesh, owner=own[order].astype(np.int32), neighbour=nei[keep].astype(np.int32), n_cells=int(new.max()) + 1,
               face_offsets=np.concatenate([[0], np.cumsum([len(faces[f]) for f in order])]).astype(np.int32),
               face_verts=np.concatenate([faces[f] for f in order]).astype(np.int32),
               patches=[dict(p, startFace=p["startFace"] - nI + len(keep)) for p in mesh["patches"]])
    return out


def _case(name):
    from dugksfoam_gb300 import cases

    dim, run, nxi = name.split("-")
    gas, rho0 = cases.gas_from_kn(0.1)
    if dim == "2d":
        mesh, two_d = merged(cases.structured_mesh(12, 9, 1, two_d=True), 12, int(run)), True
    else:
        mesh, two_d = merged(cases.structured_mesh(6, 5, 4, lz=1.0, two_d=False), 6, int(run)), False
    return cases.make_case(mesh, gas, rho0, int(nxi), 4.0 * np.sqrt(2 * gas["R"] * 273.0), two_d=two_d)


@pytest.mark.parametrize("name", ["2d-2-8", "2d-3-9", "2d-2-13", "2d-3-14", "3d-2-6", "3d-3-8", "3d-3-5"])
def test_merged_cells_match_oracle(built_lib, oracle_lib, name):
    from dugksfoam_gb300 import cases, solver
    from oracle.oracle import NumpyOracle, Oracle

    case, steps = _case(name), 12
    dt = cases.stable_dt(case)
    a, b = Oracle(case), NumpyOracle(case)
    a.step(dt, steps)
    b.step(dt, steps)
    want, other = a.cell(), b.cell()
    for prec in (solver.FP64, solver.FP32_FP64MOM):
        s = solver.FvDVM(case, precision=prec)
        s.set_dt(dt)
        s.evolution(steps)
        got = s.macros()
        s.close()
        for k in FIELDS:
            floor = rel_err(other[k], want[k])
            e = rel_err(got[k], want[k])
            for j in range(2):
                tol = 1e-5 if prec == solver.FP32_FP64MOM else max(1e-12, 4 * floor[j])
                assert e[j] <= tol, (name, prec, k, e, floor)
