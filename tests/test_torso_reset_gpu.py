"""hp_torso_reset has forgotten the last frame when it returns, whatever the
default stream is at work on: solves run on a stream that does not wait for it."""
import numpy as np
import pytest

from tests.test_pcg_resident_gpu import _box

pytestmark = pytest.mark.gpu


def test_reset_behind_work_on_the_default_stream():
    import torch
    solver, *_ = _box((40, 34, 44), seed=3)
    vm = np.array([-80.0, 20.0], np.float32)
    try:
        want, st = solver.solve_frame(vm, 1e-4, "rel", 4000)
        assert st.iterations > 0
        a = torch.randn(4096, 4096, device="cuda")
        for _ in range(40):                 # some milliseconds of work
            a = torch.tanh(a @ a)
        solver.reset()
        out, st2 = solver.solve_frame(vm, 1e-4, "rel", 4000)
        assert st2.iterations == st.iterations
        np.testing.assert_array_equal(out, want)
    finally:
        solver.close()
