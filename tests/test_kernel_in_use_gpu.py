"""hp_mono_kernel_info names the kernel that advances the steps."""
import dataclasses

import pytest

from tests import cases

pytestmark = pytest.mark.gpu

SPLIT, RESIDENT = 3, 4


def _kernel(prob, kernel):
    from hrdayapy_b200 import monodomain as M
    sim = M.MonoHandle(dataclasses.replace(prob, kernel=kernel))
    info = sim.kernel_info()
    sim.close()
    return info


def _slab(shape, theta=0.0):
    from hrdayapy_b200 import monodomain as M
    from hrdayapy_b200 import synthetic
    (nodes, el, act, S, phi), _, kw = synthetic.slab(*shape)
    return M.prepare(nodes, el, act, S, S, phi, theta=theta, cg_tol=1e-6, **dict(kw, T=2.0))[0]


def _ragged(shape, theta=0.0):
    from hrdayapy_b200 import monodomain as M
    args, fibre, kw = cases.ragged_aniso_case(shape=shape, T=1.0)
    nodes, el, act, S, phi = args
    return M.prepare(nodes, el, act, S, S, phi, fibre_dir=fibre, anisotropic=True, theta=theta,
                     **dict(kw, A_P=2.0 / kw["R_P"]))[0]


@pytest.mark.parametrize("make, size, theta, auto", [
    (_slab, (1, 1, 1), 0.0, RESIDENT), (_slab, (33, 17, 19), 0.0, RESIDENT),
    (_slab, (64, 64, 16), 0.0, RESIDENT), (_slab, (64, 64, 17), 0.0, SPLIT),
    (_slab, (64, 64, 17), 0.5, RESIDENT), (_ragged, (28, 24, 18), 0.0, RESIDENT),
    (_ragged, (28, 24, 18), 0.5, RESIDENT), (_ragged, (62, 60, 58), 0.0, RESIDENT),
    (_ragged, (80, 76, 72), 0.0, SPLIT), (_ragged, (80, 76, 72), 0.5, SPLIT)])
def test_auto_is_resident_where_the_heart_fits(make, size, theta, auto):
    prob = make(size, theta)
    kernel, grid, smem = _kernel(prob, 0)
    assert kernel == auto
    if auto == RESIDENT:
        # one thread a cell in blocks of 64 to 640, one block a multiprocessor at most
        cells = prob.n_myo + prob.n_pk
        assert grid * 640 >= cells and 0 < smem and grid <= max(1, (cells + 95) // 64, 148)
    assert _kernel(prob, 3)[0] == SPLIT


def test_resident_is_not_a_kernel_to_ask_for():
    from hrdayapy_b200 import _lib
    with pytest.raises((ValueError, _lib.HpError)):
        _kernel(_slab((8, 8, 8)), RESIDENT)


def test_tuned_small_heart_stays_resident():
    """The resident steps take less than half a split step's time at this size."""
    from hrdayapy_b200 import monodomain as M
    from hrdayapy_b200.autotune import tune
    best, table = tune(_ragged((28, 24, 18)), steps=200, warmup=20)
    sim = M.MonoHandle(best)
    assert sim.kernel_info()[0] == RESIDENT, table
    sim.close()
