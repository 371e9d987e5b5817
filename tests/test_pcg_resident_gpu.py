"""The resident PCG launch over the sizes where it changes shape: one cell to
a few cells, odd and even padded rows, short and long lines, and blocks that
keep all vectors, the residual alone or nothing in shared memory."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _box(shape, seed=0, materials=3):
    """A tissue box of random material slabs, a dipole source in its middle."""
    from hrdayapy_b200.ecg import torso as T
    rng = np.random.default_rng(seed)
    lab = np.ones(shape, np.uint8)
    for ax in range(3):
        cut = rng.integers(0, shape[ax], 2)
        sl = [slice(None)] * 3
        sl[ax] = slice(cut.min(), cut.max())
        lab[tuple(sl)] = 1 + rng.integers(0, materials)
    if min(shape) >= 6:            # air: ragged line ends, a hole inside the lines
        lab[:2, :2, :] = 0
        lab[:, -1, : shape[2] // 3] = 0
        lab[shape[0] // 2, shape[1] // 2, shape[2] // 2] = 0
    table = np.concatenate([[0.0], rng.uniform(0.05, 0.7, materials)])
    rows = np.flatnonzero(lab.ravel())
    pair = np.array([[0, 0, 0], [0, 0, 1]])
    proj = np.array([len(rows) // 3, 2 * len(rows) // 3], np.int32)
    solver = T.TorsoSolver(lab, table, 1.5, len(rows) // 2, T.heart_neighbours(pair), proj, 0.2625,
                           0.4, np.arange(len(rows)))
    return solver, lab, table, rows


def _dense(lab, table, rows, pin):
    n = len(rows)
    index = -np.ones(lab.size, np.int64)
    index[rows] = np.arange(n)
    A = np.zeros((n, n))
    ijk = np.stack(np.unravel_index(rows, lab.shape), 1)
    for ax in range(3):
        up = ijk.copy()
        up[:, ax] += 1
        ok = up[:, ax] < lab.shape[ax]
        a = np.flatnonzero(ok)
        b = index[np.ravel_multi_index(up[ok].T, lab.shape)]
        a, b = a[b >= 0], b[b >= 0]
        sa, sb = table[lab.ravel()[rows[a]]], table[lab.ravel()[rows[b]]]
        g = 2 * sa * sb / (sa + sb) / 1.5e-3 ** 2
        np.add.at(A, (a, a), g)
        np.add.at(A, (b, b), g)
        np.add.at(A, (a, b), -g)
        np.add.at(A, (b, a), -g)
    A[pin] = 0.0
    A[:, pin] = 0.0
    A[pin, pin] = 1.0
    return A


@pytest.mark.parametrize("shape", [(1, 1, 2), (2, 1, 3), (3, 4, 5), (7, 6, 31), (6, 7, 32), (6, 8, 33),
                                   (8, 7, 64), (7, 9, 65)])
def test_small_boxes_vs_dense_fp64(shape):
    solver, lab, table, rows = _box(shape, seed=sum(shape))
    try:
        vm = np.array([-80.0, 20.0], np.float32)
        for rule, tol in (("rel", 1e-6), ("rms", 1e-4), ("linf", 1e-4), ("p99", 1e-4)):
            solver.reset()
            out, st = solver.solve_frame(vm, tol, rule, 3000)
            x, b = solver.solution(), solver.rhs().astype(np.float64)
            A = _dense(lab, table, rows, len(rows) // 2)
            res = np.linalg.norm(b - A @ x) / max(np.linalg.norm(b), 1e-300)
            if rule == "rel":
                assert st.status == 0 and res <= 1.05e-6
            elif st.status == 0:
                z = np.abs((b - A @ x) / np.diag(A)) * 1e3
                z[len(rows) // 2] = 0.0
                stat = {"rms": np.sqrt(np.mean(z ** 2)), "linf": z.max(),
                        "p99": np.quantile(z, 0.99)}[rule]
                # FP32 residual against FP64: z carries about 1e-6 of the potentials
                assert stat <= tol + 1e-5 * max(1.0, np.abs(x).max() * 1e3)
            np.testing.assert_allclose(out, (x * 1e3).astype(np.float32), rtol=1e-6, atol=1e-9)
    finally:
        solver.close()


@pytest.mark.parametrize("shape", [(125, 121, 130), (120, 118, 131), (205, 200, 201)])
def test_large_boxes_reach_the_true_residual(shape):
    """About 1.9 M cells (the residual in shared memory) and 8.2 M (nothing);
    the FP64 true residual is evaluated by a kernel of its own."""
    solver, *_ = _box(shape, seed=3)
    try:
        vm = np.array([-80.0, 20.0], np.float32)
        out, st = solver.solve_frame(vm, 1e-4, "rel", 4000)
        assert st.status == 0 and 0.0 < st.rel_residual <= 1e-4
        again, st2 = solver.solve_frame(vm, 1e-4, "rel", 4000)   # warm start: nothing left to do
        assert st2.iterations == 0
        np.testing.assert_array_equal(out, again)
    finally:
        solver.close()
