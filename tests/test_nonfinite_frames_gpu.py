"""A frame with a NaN, an infinity or an overflow is an error of that frame
alone: the next frame is solved as by a fresh handle."""
import contextlib

import numpy as np
import pytest

from tests.test_pcg_resident_gpu import _box

pytestmark = pytest.mark.gpu

VM = np.array([-80.0, 20.0], np.float32)
BAD = [np.nan, np.inf, 3e38]


@pytest.mark.parametrize("bad", BAD)
@pytest.mark.parametrize("rule", ["rel", "rms", "linf", "p99"])
@pytest.mark.parametrize("shape", [(9, 8, 64), (9, 8, 65), (125, 121, 130)])
def test_torso_recovers_after_a_bad_frame(shape, rule, bad):
    from hrdayapy_b200 import _lib
    tol = 1e-4
    fresh, *_ = _box(shape, seed=3)
    want, st = fresh.solve_frame(VM, tol, rule, 4000)
    fresh.close()
    assert st.status == 0
    solver, *_ = _box(shape, seed=3)
    try:
        with pytest.raises(_lib.HpError):
            solver.solve_frame(np.array([bad, -bad], np.float32), tol, rule, 4000)
        out, st2 = solver.solve_frame(VM, tol, rule, 4000)
        assert st2.status == 0 and st2.iterations == st.iterations
        np.testing.assert_array_equal(out, want)
    finally:
        solver.close()


@pytest.mark.parametrize("bad", BAD)
def test_flexible_cg_recovers_after_a_bad_frame(bad):
    from hrdayapy_b200 import _lib
    from hrdayapy_b200.ecg.precond import LearnedPreconditioner
    from tests.test_precond_gpu import _small, _wave_frames
    solver, grid, labels, table, dx, vox = _small(shape=(16, 24, 256))
    pc = LearnedPreconditioner(solver, labels, len(table), coarse_agg=8)
    try:
        vm = _wave_frames(vox, 3, 1)[1]
        want, st = pc.solve_frame(vm, 1e-6, use_net=False)
        assert st.status == 0 and st.restarts == 0
        solver.reset()
        broken = vm.copy()
        broken[len(vm) // 2:len(vm) // 2 + 2] = bad, -bad
        with contextlib.suppress(_lib.HpError):
            pc.solve_frame(broken, 1e-6, use_net=False)
        out, st2 = pc.solve_frame(vm, 1e-6, use_net=False)
        assert (st2.status, st2.iterations, st2.restarts) == (0, st.iterations, 0)
        np.testing.assert_array_equal(out, want)
    finally:
        pc.close()
        solver.close()
