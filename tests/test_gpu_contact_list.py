"""The candidate list that stays while the nodes have used up less than half of
its room: it is kept over several lifetimes of a slow motion, and built anew when a
new state puts the nodes elsewhere.  Closed pairs and states against the oracle's
every-step search."""
import numpy as np
import pytest

import contact_cases as cc
from dynlattice_b200.abi import DL_PLAIN_FP64
from dynlattice_b200.engine import Lattice
from helpers import rel_err
from oracle_ffi import Oracle

pytestmark = pytest.mark.gpu


def test_list_is_kept_while_it_covers_the_motion(gpu):
    spec = cc.cross(gap0=0.02e-3)
    v0 = np.zeros((spec.n_nodes, 6))
    v0[spec.rod_nodes[1], 2] = -2.0
    o, g = Oracle(spec), Lattice(spec, DL_PLAIN_FP64)
    o.set_state(v=v0)
    g.set_state(v=v0)
    # 30 um at 2 m/s: lifetimes of 25 um x 1/4, x 3/16, x 9/64 fit one list (half
    # margin 100 um, kept below 50 um)
    o.run(1500)
    g.run(1500)
    assert g.contact_stats()[1] == 1
    po, _ = o.contact_pairs()
    pg, _ = g.contact_pairs()
    assert po.shape[0] > 0 and np.array_equal(po, pg)
    assert rel_err(g.state()[0], o.state()[0]) < 1e-9
    assert g.error_word() == 0


def test_new_state_elsewhere_builds_anew(gpu):
    spec = cc.cross(gap0=1.0e-3)  # far apart: no candidate
    g = Lattice(spec, DL_PLAIN_FP64)
    g.run(3)
    assert g.contact_stats()[0] == 0
    u = cc.shift_rod(spec, 1, (0, 0, -1.02e-3))
    o = Oracle(spec)
    o.set_state(u=u)
    g.set_state(u=u, v=np.zeros((spec.n_nodes, 6)), theta=np.zeros((spec.n_nodes, 3)))
    o.run(1)
    g.run(1)
    po, _ = o.contact_pairs()
    pg, _ = g.contact_pairs()
    assert po.shape[0] == 1 and np.array_equal(po, pg)
