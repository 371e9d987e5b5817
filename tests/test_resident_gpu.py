"""The resident step kernel (kernel AUTO on a heart that fits on the chip)
against the split step: the explicit step bit for bit, the theta-scheme (the
same CG with its sums in another order) to rounding."""
import dataclasses

import numpy as np
import pytest

from tests import cases
from tests.test_theta_gpu import _run_theta

pytestmark = pytest.mark.gpu


def _explicit(prob, kernel, runs):
    from hrdayapy_b200 import monodomain as M
    sim = M.MonoHandle(dataclasses.replace(prob, kernel=kernel))
    for n in runs:
        sim.run(n)
    out = (sim.vm_frames(), *sim.anim_frames(), *sim.events(), *sim.voltage(), *sim.state())
    assert sim.steps_done == sum(runs)
    sim.close()
    return out


def _compare(prob, runs):
    a, b = _explicit(prob, 0, runs), _explicit(prob, 3, runs)
    for x, y in zip(a, b):
        np.testing.assert_array_equal(x, y)


@pytest.mark.parametrize("brick", [(4, 4, 8), (4, 8, 8), (2, 4, 16), (8, 8, 8)])
def test_resident_equals_split_on_ragged_heart(brick):
    """19-point operator, tree and junctions, snapshots and animation frames
    that do not line up with the runs; runs of one and three steps take the
    split kernels on the same handle."""
    from hrdayapy_b200 import monodomain as M
    args, fibre, kw = cases.ragged_aniso_case(T=3.0)
    nodes, el, act, S, phi = args
    prob, _ = M.prepare(nodes, el, act, S, S, phi, fibre_dir=fibre, anisotropic=True,
                        vm_save_dt=0.14, save_every=11, act_threshold=-20.0,
                        deact_threshold=-20.0, brick=brick, **dict(kw, A_P=2.0 / kw["R_P"]))
    _compare(prob, (1, 4, 3, 50, 7, 85))


@pytest.mark.parametrize("shape", [(1, 1, 1), (3, 2, 1), (5, 7, 9), (33, 17, 19), (64, 64, 16), (64, 64, 17)])
def test_resident_equals_split_on_slabs(shape):
    """7-point operator from one cell to one beyond the resident range."""
    from hrdayapy_b200 import monodomain as M
    from hrdayapy_b200 import synthetic
    args, _, kw = synthetic.slab(*shape)
    nodes, el, act, S, phi = args
    prob, _ = M.prepare(nodes, el, act, S, S, phi, vm_save_dt=0.1, **dict(kw, T=2.0))
    _compare(prob, (37, 63))


def test_resident_equals_split_with_wide_blocks():
    """19-point operator on more cells than 448 threads a block hold."""
    from hrdayapy_b200 import monodomain as M
    args, fibre, kw = cases.ragged_aniso_case(shape=(62, 60, 58), T=1.0)
    nodes, el, act, S, phi = args
    prob, _ = M.prepare(nodes, el, act, S, S, phi, fibre_dir=fibre, anisotropic=True,
                        vm_save_dt=0.2, **dict(kw, A_P=2.0 / kw["R_P"]))
    assert 148 * 448 < prob.n_myo < 148 * 640
    _compare(prob, (20, 30))


@pytest.mark.parametrize("theta", [0.5, 1.0])
@pytest.mark.parametrize("aniso", [False, True])
def test_resident_theta_matches_tiled_passes(theta, aniso):
    if aniso:
        args, fibre, kw = cases.ragged_aniso_case(T=6.0)
    else:
        args, kw = cases.iso_case()
        kw, fibre = dict(kw, T=6.0), None
    import hrdayapy_b200.monodomain as M
    a = _run_theta(args, kw, fibre=fibre, theta=theta)
    keep = M.MonoHandle.__init__

    def split(self, prob, stream=None):
        keep(self, dataclasses.replace(prob, kernel=3), stream)

    M.MonoHandle.__init__ = split
    try:
        b = _run_theta(args, kw, fibre=fibre, theta=theta)
    finally:
        M.MonoHandle.__init__ = keep
    assert a[4][1:] == b[4][1:]                       # solves, unconverged, breakdowns
    assert abs(a[4][0] - b[4][0]) <= 0.01 * b[4][0]    # a residual at the threshold may tip over
    # each solve stops at ||r|| <= 1e-6 ||rhs||: per cell at most 1e-6 sqrt(N) 90 mV a step
    bound = 1e-6 * np.sqrt(a[1].shape[1]) * 90.0 * 10.0
    assert np.abs(a[1] - b[1]).max() <= bound
    np.testing.assert_array_equal(a[3], b[3])
