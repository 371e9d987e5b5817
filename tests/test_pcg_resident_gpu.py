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


@pytest.mark.parametrize("agg", [-1, 4, 8, 16, 32, 64])
def test_flexible_cg_takes_the_steps_of_a_host_loop(agg):
    """The flexible CG forms z = M(r) inside its passes, from segment sums of
    r; a host loop in FP64 around the preconditioner's own apply (z stored)
    must take the same number of iterations for every aggregate edge."""
    import torch
    from tests.test_precond_gpu import _small, _wave_frames
    from hrdayapy_b200.ecg.precond import LearnedPreconditioner
    solver, grid, labels, table, dx, vox = _small(shape=(16, 24, 256))
    pc = LearnedPreconditioner(solver, labels, len(table), coarse_agg=agg)
    try:
        vm = _wave_frames(vox, 3, 1)[1]
        out, st = pc.solve_frame(vm, 1e-6, use_net=False)
        assert st.status == 0 and st.rel_residual <= 1e-6 and st.restarts == 0
        lab = torch.nn.functional.pad(torch.as_tensor(labels).long(), (1,) * 6).cuda()
        sig = torch.as_tensor(table, dtype=torch.float64).cuda()[lab]
        pin = int(pc.arrays.pin_cell)
        faces = []
        for ax in range(3):
            a, b = sig.narrow(ax, 0, sig.shape[ax] - 1), sig.narrow(ax, 1, sig.shape[ax] - 1)
            faces.append(torch.where((a > 0) & (b > 0), 2 * a * b / (a + b).clamp(min=1e-30), 0 * a)
                         / (dx * 1e-3) ** 2)

        def A(x):
            y = torch.zeros_like(x)
            for ax, w in enumerate(faces):
                n = x.shape[ax]
                f = w * (x.narrow(ax, 0, n - 1) - x.narrow(ax, 1, n - 1))
                y.narrow(ax, 0, n - 1).add_(f)
                y.narrow(ax, 1, n - 1).sub_(f)
            y.view(-1)[pin] = 0.0
            return y

        def M(r):
            r32 = r.float().contiguous()
            z = torch.zeros_like(r32)
            torch.cuda.synchronize()
            pc.apply(r32.data_ptr(), z.data_ptr(), use_net=False)
            torch.cuda.synchronize()
            return z.double()

        b = torch.zeros_like(sig)
        b[lab > 0] = torch.as_tensor(solver.rhs(), dtype=torch.float64).cuda()
        r, its = b.clone(), 0
        z = M(r)
        p = z.clone()
        while torch.linalg.norm(r) >= 0.5e-6 * torch.linalg.norm(b) and its < 1000:
            q = A(p)
            pq = torch.sum(p * q)
            r = r - torch.sum(p * r) / pq * q
            z = M(r)
            p = z - torch.sum(z * q) / pq * p
            its += 1
        # FP32 vectors against FP64 ones: a few per cent of the iterations
        assert abs(its - st.iterations) <= 2 + 0.05 * its, (its, st.iterations)
    finally:
        pc.close()
        solver.close()
