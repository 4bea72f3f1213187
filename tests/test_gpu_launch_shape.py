"""The kernel and launch shape that dl_run takes (dl_get_launch_shape): what the
autotuner keeps, and which models run in the one-barrier kernel."""
import pytest

from dynlattice_b200 import lattices
from dynlattice_b200.abi import DL_MIXED
from dynlattice_b200.engine import Lattice

pytestmark = pytest.mark.gpu


def test_autotune_can_keep_the_automatic_shape(gpu):
    """On a 4^3 BCC lattice the automatic shape is the one-barrier kernel, half as
    long a step as any shape with a thread count set by hand."""
    g = Lattice(lattices.lattice_impact("bcc", n=4), DL_MIXED)
    assert g.launch_shape(100)["kernel"] == "one_barrier"
    mode, threads, _ = g.autotune(100)
    assert (mode, threads) == (0, 0)
    assert g.launch_shape(100)["kernel"] == "one_barrier"
    g.set_launch_shape(0, 128)
    assert g.launch_shape(100)["kernel"] == "two_barriers"
    assert g.launch_shape(100)["threads"] == 128
    g.set_launch_shape(1, 0)
    assert g.launch_shape(100)["kernel"] == "two_launches"
