"""The FP32 face sweep starts beside the cell gather of the step before: many
steps in one go give bit for bit what the same steps give with the GPU waited
for after each (no overlap), also where boundary kernels follow the gather."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name", ["quads", "quads_many_tiles", "hexes", "channel"])
def test_overlapped_steps_equal_separate_steps(built_lib, monkeypatch, name):
    from dugksfoam_gb300 import cases, solver

    if name == "quads_many_tiles":
        monkeypatch.setenv("DUGKS_TILE_CELLS", "6")
    case = {"hexes": lambda: cases.cavity3d(n=8, nxi=8), "channel": lambda: cases.channel2d(nx=30, ny=14, nxi=12)}.get(
        name, lambda: cases.cavity2d(n=40, nxi=16))()
    out = []
    for split in (False, True):
        s = solver.FvDVM(case, precision=solver.FP32_FP64MOM)
        s.set_dt(cases.stable_dt(case))
        for n in [1] * 60 if split else [60]:
            s.evolution(n)
            s.synchronize()
        out.append(s.macros())
        s.close()
    for k in ("rho", "U", "T", "q"):
        assert np.array_equal(out[0][k], out[1][k]), (name, k)
