"""The one-barrier kernel's share-out: made by the first run that can use it, left
out for models that the kernel cannot hold, and the same bits as the two-barrier kernels
over its ragged and two-block forms (each case states the launch it expects)."""
import numpy as np
import pytest
import torch

from dynlattice_b200 import lattices
from dynlattice_b200.abi import DL_MIXED, DL_PLAIN_FP64
from dynlattice_b200.engine import Lattice

pytestmark = pytest.mark.gpu


def _free():
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def test_runs_take_no_device_memory(gpu):
    """The share-out is made by the first run of several steps, in memory that the
    handle has; a run of another kind before it does not make it."""
    spec = lattices.lattice_impact("bcc", n=20)
    Lattice(spec, DL_PLAIN_FP64).run(2)   # loads the kernels
    g = Lattice(spec, DL_PLAIN_FP64)
    g.set_group_output(True)
    g.run(1)
    g.run(3)
    g.set_group_output(False)
    before = _free()
    assert g.launch_shape(2)["kernel"] == "one_barrier"
    for n in (1, 2, 3):
        g.run(n)
    g.synchronize()
    assert _free() == before


# topology, cells, elements per strut, Gauss points, plastic, precision; blocks
# (148 SMs: more than 148 are two per SM), element records in shared memory
FORMS = [
    ("sc", 22, 3, 1, False, DL_MIXED, 291, False),       # two per SM, ragged
    ("sc", 22, 3, 1, False, DL_PLAIN_FP64, 291, False),
    ("bcc", 20, 2, 2, True, DL_MIXED, 291, False),       # two per SM, FP32 return map inline
    ("bcc", 14, 2, 2, True, DL_MIXED, 145, True),        # one per SM, records beside the copies
    ("bcc", 14, 2, 2, True, DL_PLAIN_FP64, 289, False),
    ("bcc", 3, 2, 2, True, DL_MIXED, 14, True),          # 432 elements in blocks of 32
    ("bcc", 3, 1, 2, True, DL_PLAIN_FP64, 1, True),      # one block
]


def _spec(topology, n, per_strut, gauss, plastic):
    return lattices.lattice_impact(topology, n=n, elems_per_strut=per_strut, n_gauss=gauss, plastic=plastic,
                                   velocity=50.0, seed=n)


@pytest.mark.parametrize("topology,n,per_strut,gauss,plastic,precision,blocks,records", FORMS)
def test_one_barrier_forms(gpu, topology, n, per_strut, gauss, plastic, precision, blocks, records):
    spec = _spec(topology, n, per_strut, gauss, plastic)
    rng = np.random.default_rng(n)
    u = rng.normal(scale=1e-6, size=(spec.n_nodes, 3))
    th = rng.normal(scale=1e-3, size=(spec.n_nodes, 3))
    one, two = Lattice(spec, precision), Lattice(spec, precision)
    two.set_launch_shape(0, 128)
    shape = one.launch_shape(9)
    copy = 252 if precision == DL_MIXED else 300  # bytes of a node copy; the rest are records
    assert (shape["kernel"], shape["blocks"]) == ("one_barrier", blocks)
    assert ((shape["shared_bytes"] - 16) % copy != 0) == records
    assert two.launch_shape(9)["kernel"] == "two_barriers"
    for g in (one, two):
        g.set_state(u=u, theta=th)
        for k in (9, 2, 25):
            g.run(k)
        g.synchronize()
    for a, b in zip(one.state(), two.state()):
        assert np.array_equal(a, b)
    if plastic:
        for a, b in zip(one.history(), two.history()):
            assert np.array_equal(a, b)
    assert one.error_word() == two.error_word() == 0


@pytest.mark.parametrize("topology,n,per_strut,gauss,plastic,precision", [
    ("sc", 25, 3, 1, False, DL_MIXED),          # 118,976 nodes: the copies do not fit
    ("sc", 25, 3, 1, False, DL_PLAIN_FP64),
    ("bcc", 21, 2, 2, True, DL_PLAIN_FP64),     # 93,997 nodes: no longer FP64
])
def test_models_too_large_for_the_copies(gpu, topology, n, per_strut, gauss, plastic, precision):
    g = Lattice(_spec(topology, n, per_strut, gauss, plastic), precision)
    assert g.launch_shape(9)["kernel"] == "two_barriers"
    assert g.launch_shape(1)["kernel"] == "one_step"


def test_features_of_the_extended_kernels(gpu):
    g = Lattice(_spec("bcc", 3, 2, 2, True), DL_MIXED)
    assert g.launch_shape(1)["kernel"] == "one_step"
    g.set_group_output(True)
    assert g.launch_shape(9)["kernel"] == "two_barriers_x"
    g.set_group_output(False)
    assert g.launch_shape(9)["kernel"] == "one_barrier"
