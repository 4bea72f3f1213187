"""The one-barrier kernel's share-out is made by the first run that can use it."""
import pytest
import torch

from dynlattice_b200 import lattices
from dynlattice_b200.abi import DL_PLAIN_FP64
from dynlattice_b200.engine import Lattice

pytestmark = pytest.mark.gpu


def _free():
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def test_share_out_is_made_by_the_run_that_uses_it(gpu):
    """A handle that is stepped one by one holds one set of end-force slots; the
    first run of several steps brings the second one."""
    spec = lattices.lattice_impact("bcc", n=20)
    slots = spec.n_elems * 12 * 8
    g = Lattice(spec, DL_PLAIN_FP64)
    g.run(1)
    g.set_group_output(True)   # the extended kernels: no share-out either
    g.run(3)
    g.set_group_output(False)
    g.run(1)
    g.synchronize()
    before = _free()
    g.run(2)
    g.synchronize()
    used = before - _free()
    assert used >= slots
    g.run(3)
    g.synchronize()
    assert before - _free() == used
