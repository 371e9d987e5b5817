"""Flexible CG with aggregates of edge 1 and 2: every iteration applies the M
that hp_precond_apply gives."""
import numpy as np
import pytest

import tests.test_precond_gpu as P
from tests.test_pcg_resident_gpu import test_flexible_cg_takes_the_steps_of_a_host_loop as host_loop

pytestmark = pytest.mark.gpu


def _little_tissue(shape):
    """At most HP_PC_MAX_COARSE = 2,048 tissue cells in a box of (8, 8, 256)."""
    from hrdayapy_b200.ecg import torso as T
    lab = np.zeros((8, 8, 256), np.uint8)
    lab[1:7, 1:7, 3:59] = 1
    lab[3:5, 2:6, 20:40] = 2
    rows = np.flatnonzero(lab.ravel())
    table = np.array([0.0, 0.2, 0.6])
    vox = np.argwhere(np.ones((4, 4, 40), bool))
    at = vox + [2, 2, 10]
    proj = np.searchsorted(rows, np.ravel_multi_index(at.T, lab.shape)).astype(np.int32)
    solver = T.TorsoSolver(lab, table, 1.5, len(rows) // 2, T.heart_neighbours(vox), proj, 0.2625,
                           1.5, np.arange(len(rows)))
    return solver, None, lab, table, 1.5, vox


@pytest.mark.parametrize("agg", [1, 2])
def test_small_aggregates_take_the_steps_of_a_host_loop(agg, monkeypatch):
    small = P._small
    monkeypatch.setattr(P, "_small", _little_tissue if agg == 1
                        else lambda shape: small(shape=(8, 8, 256)))
    host_loop(agg)
