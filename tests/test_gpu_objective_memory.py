"""What objective calls keep on the device: counted in device_bytes, the same
numbers from kept buffers as from a new handle's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _handle():
    from dugksfoam_gb300 import cases, solver

    s = solver.FvDVM(cases.cavity2d(n=6, nxi=8), precision=solver.FP64)
    s.set_dt(cases.case_dt(cases.cavity2d(n=6, nxi=8)))
    return s


def test_device_bytes_count_what_calls_keep(built_lib):
    import torch

    s = _handle()
    o = dict(n_steps=3, avg_first=1, q_patch=0, stress_patch=1, checkpoint_every=2)
    s.objective_adjoint(**o)  # loads the kernels
    s.close()
    s = _handle()
    b0, f0 = s.info()["device_bytes"], torch.cuda.mem_get_info()[0]
    s.objective_adjoint(**o)
    b1, f1 = s.info()["device_bytes"], torch.cuda.mem_get_info()[0]
    assert b1 - b0 == f0 - f1 and b1 > b0  # whole chunks of 64 MB
    s.objective_value(**{k: o[k] for k in o if k != "checkpoint_every"})
    assert s.info()["device_bytes"] == b1
    s.close()
    assert torch.cuda.mem_get_info()[0] >= f0


def test_calls_of_other_sizes_on_kept_buffers(built_lib):
    base = dict(avg_first=1, q_patch=0, stress_patch=1)
    adj = [dict(base, n_steps=n, checkpoint_every=k) for n, k in ((40, 40), (3, 2), (40, 7), (9, 100))]
    d = np.random.default_rng(0).standard_normal(_handle().info()["n_wall_faces"])

    def calls(new):
        s = _handle()
        for o in adj:
            v = {k: o[k] for k in o if k != "checkpoint_every"}
            for f in (lambda: s.objective_adjoint(**o), lambda: s.objective_value(**v),
                      lambda: s.objective_tangent(d, 0.7, **v)):
                if new:
                    s.close()
                    s = _handle()
                yield f()
        s.close()

    for a, b in zip(calls(False), calls(True)):
        for x, y in zip(np.atleast_1d(np.asarray(a, object)), np.atleast_1d(np.asarray(b, object))):
            assert np.array_equal(x, y)
