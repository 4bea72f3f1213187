"""Models that run in one block (its own barrier in place of the grid's)
against the oracle and against the launch over several blocks, at the edges:
the last size of one block, the first of several, and sizes around the
block's 128 threads."""
import numpy as np
import pytest

from dynlattice_b200 import lattices
from dynlattice_b200.abi import DL_PLAIN_FP64
from dynlattice_b200.engine import Lattice
from helpers import rel_err
from oracle_ffi import Oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_elems", [1, 31, 32, 127, 128, 255, 256])
def test_rod_in_one_block(gpu, n_elems):
    spec = lattices.straight_rod(n_elems, length=n_elems / 32.0, tip_force=1e3, ramp_steps=50)
    o = Oracle(spec)
    one = Lattice(spec, DL_PLAIN_FP64)
    many = Lattice(spec, DL_PLAIN_FP64)
    many.set_launch_shape(0, 32)
    tip = spec.groups["free"]
    for g in (one, many):
        g.set_sampling(7, tip, 20)
        g.run(100)
        g.synchronize()
    o.run(100)
    uo = o.state()[0]
    (u1, t1, v1), (u2, t2, v2) = one.state(), many.state()
    # the same arithmetic on the same items, whatever the number of blocks
    assert np.array_equal(u1, u2) and np.array_equal(t1, t2) and np.array_equal(v1, v2)
    assert rel_err(u1, uo) < 1e-9
    s1, r1, e1 = one.samples()
    s2, r2, e2 = many.samples()
    assert np.array_equal(s1, s2) and np.array_equal(r1, r2) and s1.size == 14
    assert rel_err(e1, e2) < 1e-12
    assert one.energies()["external_work"] == pytest.approx(o.energies()["external_work"], rel=1e-9)
    assert one.error_word() == 0
