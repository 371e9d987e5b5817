"""Handles of different size alive at once: each runs as it does alone, in
both orders of creation.  They share their kernels, so nothing a handle sets
on a kernel may be sized for that handle alone."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


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
