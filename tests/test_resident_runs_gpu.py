"""Resident runs that are cut into several launches (65,536 steps each): a last
launch of one step passes no grid barrier."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(3, 2, 1), (20, 10, 48)])
@pytest.mark.parametrize("last", [1, 2])
def test_long_run_with_a_short_last_launch(shape, last):
    """On one and on about a hundred blocks: as the same steps in launches that all pass
    barriers, at the end and four steps on."""
    from hrdayapy_b200 import monodomain as M
    from hrdayapy_b200 import synthetic
    (nodes, el, act, S, phi), _, kw = synthetic.slab(*shape)
    n = (1 << 16) + last
    prob, _ = M.prepare(nodes, el, act, S, S, phi, **dict(kw, T=(n + 8) * kw["dt"]))
    out = []
    for runs in ((n,), (n - 8, 8)):
        sim = M.MonoHandle(prob)
        for k in runs:
            sim.run(k)
        assert sim.steps_done == n
        now = sim.voltage()
        sim.run(4)
        out.append((*now, *sim.voltage(), *sim.state(), *sim.events()))
        sim.close()
    for a, b in zip(*out):
        np.testing.assert_array_equal(a, b)
