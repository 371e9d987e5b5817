"""The tiled step kernels' launch forms on hearts that AUTO would run resident
(kernel SPLIT): replayed graphs against direct launches, and solve loops on
the device against loops tested by the host."""
import dataclasses

import numpy as np
import pytest

from tests import cases

pytestmark = pytest.mark.gpu


def _runs(theta, chunks, cg_max_iter=100):
    from hrdayapy_b200 import monodomain as M
    args, fibre, kw = cases.ragged_aniso_case(T=4.0)
    nodes, el, act, S, phi = args
    prob, _ = M.prepare(nodes, el, act, S, S, phi, fibre_dir=fibre, anisotropic=True, theta=theta,
                        cg_tol=1e-6, cg_max_iter=cg_max_iter, vm_save_dt=kw["dt"],
                        **dict(kw, A_P=2.0 / kw["R_P"]))
    out = []
    for chunk in chunks:
        sim = M.MonoHandle(dataclasses.replace(prob, kernel=3))
        assert sim.kernel_info()[0] == 3
        half = prob.n_steps // 2 + 1
        sim.run(half, graph_chunk=chunk)
        sim.run(prob.n_steps - half, graph_chunk=chunk)
        out.append((sim.vm_frames(), *sim.voltage(), *sim.state(), np.array(sim.cn_stats())))
        sim.close()
    for other in out[1:]:
        for a, b in zip(out[0], other):
            np.testing.assert_array_equal(a, b)
    return out[0][-1]


def test_split_graph_and_direct_launch_agree():
    _runs(0.0, (0, 7, 50))


@pytest.mark.parametrize("cg_max_iter", [1, 3, 100])
def test_tiled_theta_graph_and_host_loop_agree(cg_max_iter):
    """Conditional graph nodes and the host-tested chunks run the same kernels
    in the same order, also where the iteration limit ends the loop."""
    its, solves, unconverged, _ = _runs(0.5, (0, 1, 16), cg_max_iter)
    assert its <= cg_max_iter * solves and (unconverged > 0) == (cg_max_iter < 100)


def test_counters_are_of_all_steps_enqueued():
    """cn_stats waits for the steps before it."""
    from hrdayapy_b200 import monodomain as M
    args, fibre, kw = cases.ragged_aniso_case(T=40.0)
    nodes, el, act, S, phi = args
    prob, _ = M.prepare(nodes, el, act, S, S, phi, fibre_dir=fibre, anisotropic=True, theta=0.5,
                        cg_tol=1e-6, **dict(kw, A_P=2.0 / kw["R_P"]))
    for kernel in (0, 3):
        n = prob.n_steps // 16 * 16
        sim = M.MonoHandle(dataclasses.replace(prob, kernel=kernel))
        sim.run(n, graph_chunk=16)
        assert sim.cn_stats()[1] == n
        sim.close()
