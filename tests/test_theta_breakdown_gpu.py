"""A theta-scheme solve that breaks down keeps the potential it started from,
in the tiled passes as in the resident kernel: non-finite directions never
reach it."""
import dataclasses

import numpy as np
import pytest

from tests import cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bad", [np.nan, np.inf])
@pytest.mark.parametrize("chunk", [0, 4])
def test_breakdown_keeps_the_potential(bad, chunk):
    """One non-finite face weight ends every solve before its first step (a
    breakdown, or both norms infinite); the cells beside it keep W like all
    others."""
    from hrdayapy_b200 import monodomain as M
    args, fibre, kw = cases.ragged_aniso_case(T=1.0)
    nodes, el, act, S, phi = args
    prob, _ = M.prepare(nodes, el, act, S, S, phi, fibre_dir=fibre, anisotropic=True, theta=0.5,
                        cg_tol=1e-6, vm_save_dt=kw["dt"], **dict(kw, A_P=2.0 / kw["R_P"]))
    tag = np.asarray(prob.tag).ravel()
    inner = np.flatnonzero((tag & 3 != 0) & (tag >> 2 & 63 == 63))   # all six neighbours there
    w = np.array(prob.wface, np.float32).reshape(3, -1)
    w[0, inner[len(inner) // 2]] = bad
    out = []
    for kernel in (3, 0):
        sim = M.MonoHandle(dataclasses.replace(prob, wface=w.ravel(), kernel=kernel))
        sim.run(prob.n_steps, graph_chunk=chunk)
        out.append((sim.vm_frames(), *sim.voltage(), *sim.state(), np.array(sim.cn_stats())))
        assert sim.cn_stats()[:3] == (0, prob.n_steps, 0)
        sim.close()
    assert (np.abs(out[0][0]) < 100.0).all() and (out[0][0] > -100.0).all()
    for a, b in zip(*out):
        np.testing.assert_array_equal(a, b)
