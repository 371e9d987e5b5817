"""Handles of different size alive at once: each runs as it does alone, in
both orders of creation.  They share their kernels, so nothing a handle sets
on a kernel may be sized for that handle alone."""
import numpy as np
import pytest

from tests.test_pcg_resident_gpu import _box

pytestmark = pytest.mark.gpu

VM = np.array([-80.0, 20.0], np.float32)


def _solve(solver):
    solver.reset()
    out, st = solver.solve_frame(VM, 1e-4, "rel", 4000)
    assert st.status == 0 and st.rel_residual <= 1e-4
    return out


@pytest.mark.parametrize("order", [(0, 1), (1, 0)])
@pytest.mark.parametrize("shapes", [((96, 80, 128), (40, 34, 44)), ((96, 80, 127), (40, 34, 43)),
                                    ((150, 140, 150), (125, 121, 130))])
def test_torso_handles_of_two_sizes(shapes, order):
    """Blocks that keep all vectors on the chip (even and odd padded rows), and
    the residual alone."""
    alone = []
    for shape in shapes:
        solver, *_ = _box(shape, seed=3)
        alone.append(_solve(solver))
        solver.close()
    both = {}
    try:
        for q in order:
            both[q], *_ = _box(shapes[q], seed=3)
        for q in (0, 1):
            np.testing.assert_array_equal(_solve(both[q]), alone[q])
    finally:
        for solver in both.values():
            solver.close()


def _heart(shape, theta):
    from hrdayapy_b200 import monodomain as M
    from hrdayapy_b200 import synthetic
    (nodes, el, act, S, phi), _, kw = synthetic.slab(*shape)
    prob, _ = M.prepare(nodes, el, act, S, S, phi, vm_save_dt=0.1, theta=theta, cg_tol=1e-6,
                        **dict(kw, T=1.0))
    return prob


def _run(sim):
    sim.run(sim.prob.n_steps)
    return sim.vm_frames()


@pytest.mark.parametrize("order", [(0, 1), (1, 0)])
@pytest.mark.parametrize("theta", [0.0, 0.5])
@pytest.mark.parametrize("shapes", [((48, 48, 16), (30, 20, 20)), ((64, 64, 16), (48, 48, 20))])
def test_resident_hearts_of_two_sizes(shapes, theta, order):
    """Hearts of one register budget (up to 256 and up to 448 threads a block)."""
    from hrdayapy_b200 import monodomain as M
    alone = []
    for shape in shapes:
        sim = M.MonoHandle(_heart(shape, theta))
        alone.append(_run(sim))
        sim.close()
    both = {}
    try:
        for q in order:
            both[q] = M.MonoHandle(_heart(shapes[q], theta))
        for q in (0, 1):
            np.testing.assert_array_equal(_run(both[q]), alone[q])
    finally:
        for sim in both.values():
            sim.close()
