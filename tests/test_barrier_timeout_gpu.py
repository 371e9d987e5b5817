"""A resident launch whose grid barrier gave up leaves the handle failed, and
every later call says so.  The tests mark the handle as such a launch does
(hp_mono_inject_timeout, hp_torso_inject_timeout): no wait runs out."""
import numpy as np
import pytest

from tests import cases

pytestmark = pytest.mark.gpu


def _heart(theta=0.0):
    from hrdayapy_b200 import monodomain as M
    args, fibre, kw = cases.ragged_aniso_case(T=1.0)
    nodes, el, act, S, phi = args
    prob, _ = M.prepare(nodes, el, act, S, S, phi, fibre_dir=fibre, anisotropic=True, theta=theta,
                        vm_save_dt=kw["dt"], save_every=5, **dict(kw, A_P=2.0 / kw["R_P"]))
    sim = M.MonoHandle(prob)
    sim.run(10)
    sim.vm_frames()
    return sim


CALLS = {
    "run": lambda sim: sim.run(4),
    "run_split": lambda sim: sim.run(1),
    "vm_frames": lambda sim: sim.vm_frames(0, 1),
    "vm_frames_async": lambda sim: (sim.vm_frames_async(0, 1, _pinned(sim)), sim.wait_copies()),
    "vm_frames_device": lambda sim: sim.vm_frames_device(_device(sim).data_ptr(), 0, 1),
    "anim_frames": lambda sim: sim.anim_frames(),
    "events": lambda sim: sim.events(),
    "voltage": lambda sim: sim.voltage(),
    "voltage_pk": lambda sim: _voltage_pk(sim),
    "state": lambda sim: sim.state(),
    "cn_stats": lambda sim: sim.cn_stats(),
}


def _pinned(sim):
    import torch
    return torch.empty((1, sim.prob.n_myo), dtype=torch.float32, pin_memory=True)


def _device(sim):
    import torch
    return torch.empty((1, sim.prob.n_myo), dtype=torch.float32, device="cuda")


def _voltage_pk(sim):
    from hrdayapy_b200 import _lib
    vp = np.empty(sim.prob.n_pk, np.float32)
    _lib.check(_lib.lib().hp_mono_copy_v(sim.h, None, _lib.ptr(vp), sim.stream), "hp_mono_copy_v")


@pytest.mark.parametrize("theta", [0.0, 0.5])
@pytest.mark.parametrize("call", list(CALLS))
def test_heart_calls_after_a_timeout(call, theta):
    from hrdayapy_b200 import _lib
    sim = _heart(theta)
    CALLS[call](sim)                       # in order before
    _lib.check(_lib.lib().hp_mono_inject_timeout(sim.h), "hp_mono_inject_timeout")
    done = sim.steps_done
    with pytest.raises(_lib.HpError, match="timed out"):
        CALLS[call](sim)
    assert sim.steps_done == done
    sim.close()


@pytest.mark.parametrize("launch", [1, 2, 3])
def test_training_stops_after_a_timeout(launch):
    """The launches of a training frame: the solve (one recursion at this
    tolerance), then one for each further iterate."""
    import torch
    from hrdayapy_b200 import _lib
    from hrdayapy_b200.ecg.precond import LearnedPreconditioner
    from tests.test_precond_gpu import _small, _wave_frames
    solver, grid, labels, table, dx, vox = _small(shape=(16, 24, 256))
    pc = LearnedPreconditioner(solver, labels, len(table), coarse_agg=8)
    vm = torch.from_numpy(np.ascontiguousarray(_wave_frames(vox, 3, 1)[1:2])).cuda()
    _lib.check(_lib.lib().hp_torso_inject_timeout(solver.h, launch), "hp_torso_inject_timeout")
    with pytest.raises(_lib.HpError, match="timed out"):
        pc.train(vm, ks=(4, 8), repeats=1, tol_exact=1e-2)
    pc.close()
    solver.close()


def test_a_timeout_is_of_one_handle():
    """Not of the others alive, nor of the next one made."""
    from hrdayapy_b200 import _lib
    a, b = _heart(), _heart(0.5)
    _lib.check(_lib.lib().hp_mono_inject_timeout(a.h), "hp_mono_inject_timeout")
    b.run(4)
    b.vm_frames()
    a.close()
    c = _heart()
    c.run(4)
    c.vm_frames()
    b.close()
    c.close()
