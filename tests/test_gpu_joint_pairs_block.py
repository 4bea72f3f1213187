"""Small models with many joint pairs: one block with the threads that the pairs
ask for, the same bits as several blocks, and the oracle's forces."""
import numpy as np
import pytest

import joint_cases as jc
from dynlattice_b200.abi import DL_PLAIN_FP64
from dynlattice_b200.engine import Lattice
from helpers import rel_err
from oracle_ffi import Oracle

pytestmark = pytest.mark.gpu


def _cluster(rods, margin):
    rng = np.random.default_rng(rods)
    a = rng.uniform(0.0, 0.02, (rods, 3))
    d = rng.normal(size=(rods, 3))
    d /= np.linalg.norm(d, axis=1)[:, None]
    spec = jc.rods_with_joints([(p, p + jc.L * q) for p, q in zip(a, d)], elems=1, margin=margin)
    u = np.repeat(rng.normal(scale=0.5e-3, size=(rods, 3)), 2, axis=0)  # rods shifted: joints come within 2r
    return spec, u


# threads of the block: from the items (elements, nodes, pairs), up to 128, up to
# 256 where more than 128 of them are joint pairs
@pytest.mark.parametrize("rods,margin,threads", [(3, 0.02, 32), (10, 0.1, 256), (60, 0.1, 256), (128, 0.1, 256)])
def test_block_takes_threads_for_joint_pairs(gpu, rods, margin, threads):
    spec, u = _cluster(rods, margin)
    one, many, o = Lattice(spec, DL_PLAIN_FP64), Lattice(spec, DL_PLAIN_FP64), Oracle(spec, threads=4)
    many.set_launch_shape(0, 32)
    for g in (one, many, o):
        g.set_state(u=u)
        g.run(40)
    shape = one.launch_shape(40)
    assert (shape["kernel"], shape["blocks"], shape["threads"]) == ("two_barriers_x", 1, threads)
    for x, y in zip(one.state(), many.state()):
        assert np.array_equal(x, y)
    po, _ = o.joint_contact_pairs()
    pg, _ = one.joint_contact_pairs()
    assert np.array_equal(po, pg) and (rods < 60 or po.shape[0] > 0)
    assert rel_err(one.state()[0], o.state()[0]) < 1e-9
    assert one.error_word() == 0
