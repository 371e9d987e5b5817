"""A non-finite frame is an error of the flexible CG, as of the plain PCG: not
a solve that took no iterations."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("use_net", [False, True])
@pytest.mark.parametrize("bad", [np.nan, np.inf, 3e38])
def test_bad_frame_is_an_error(bad, use_net):
    from hrdayapy_b200 import _lib
    from hrdayapy_b200.ecg.precond import LearnedPreconditioner
    from tests.test_precond_gpu import _small, _wave_frames
    solver, grid, labels, table, dx, vox = _small(shape=(16, 24, 256))
    pc = LearnedPreconditioner(solver, labels, len(table), coarse_agg=8)
    try:
        vm = _wave_frames(vox, 3, 1)[1]
        want, st = pc.solve_frame(vm, 1e-6, use_net=use_net)
        x = solver.solution()
        broken = vm.copy()
        broken[len(vm) // 2:len(vm) // 2 + 2] = bad, -bad
        with pytest.raises(_lib.HpError, match="non-finite"):
            pc.solve_frame(broken, 1e-6, use_net=use_net)
        np.testing.assert_array_equal(solver.solution(), x)   # the warm start is kept
        solver.reset()
        out, st2 = pc.solve_frame(vm, 1e-6, use_net=use_net)
        assert (st2.status, st2.iterations, st2.restarts) == (0, st.iterations, st.restarts)
        np.testing.assert_array_equal(out, want)
    finally:
        pc.close()
        solver.close()
