"""Torsos whose records of tissue lines do not fit in the blocks' shared memory
(24 bytes a line, about 1.3 M lines over the chip)."""
import numpy as np
import pytest

from tests.test_pcg_resident_gpu import _box

pytestmark = pytest.mark.gpu


def _residual(lab, table, pin_row, x, b):
    """b - A x in FP64 on a torso without air."""
    sig = table[lab]
    X = x.reshape(lab.shape)
    y = np.zeros(lab.shape)
    for ax in range(3):
        n = lab.shape[ax]
        lo, hi = np.arange(n - 1), np.arange(1, n)
        sa, sb = sig.take(lo, ax), sig.take(hi, ax)
        f = 2 * sa * sb / (sa + sb) / 1.5e-3 ** 2 * (X.take(lo, ax) - X.take(hi, ax))
        at = [slice(None)] * 3
        at[ax] = slice(0, n - 1)
        y[tuple(at)] += f
        at[ax] = slice(1, n)
        y[tuple(at)] -= f
    r = b - y.ravel()
    r[pin_row] = 0.0
    return r


@pytest.mark.parametrize("shape", [(1160, 1159, 1), (1160, 1160, 1), (1200, 1190, 2)])
def test_more_lines_than_shared_memory_holds(shape):
    """The last size whose records fit, the next one, and an even padded row."""
    solver, lab, table, rows = _box(shape, seed=5)
    vm = np.array([-80.0, 20.0], np.float32)
    try:
        out, st = solver.solve_frame(vm, 1e-3, "rel", 20000)
        assert st.status == 0 and 0.0 < st.rel_residual <= 1e-3 and st.iterations > 10
        x, b = solver.solution(), solver.rhs().astype(np.float64)
        r = _residual(lab, table, len(rows) // 2, x, b)
        # the same FP64 residual, summed in another order
        np.testing.assert_allclose(np.linalg.norm(r) / np.linalg.norm(b), st.rel_residual, rtol=1e-6)
        np.testing.assert_allclose(out, (x * 1e3).astype(np.float32), rtol=1e-6, atol=1e-9)
        solver.reset()
        for rule in ("rms", "p99"):      # one more launch shape each
            _, st = solver.solve_frame(vm, 1e-6, rule, 50)
            assert st.iterations == 50 or st.status == 0
    finally:
        solver.close()
