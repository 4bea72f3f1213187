"""The one-barrier step kernel (node copies in each block's shared memory)
against the two-barrier kernels, which run when the launch shape is set by hand:
the same arithmetic on the same items, so the same bits, over the sizes where the
share-out changes (a block per SM and two, records in shared memory or not,
remainders, one to three Gauss points, elements that flow)."""
import numpy as np
import pytest

from dynlattice_b200 import lattices
from dynlattice_b200.abi import DL_MIXED, DL_PLAIN_FP64
from dynlattice_b200.engine import Batch, Lattice

pytestmark = pytest.mark.gpu


def _spec(topology, n, per_strut, gauss, plastic):
    return lattices.lattice_impact(topology, n=n, elems_per_strut=per_strut, n_gauss=gauss, plastic=plastic,
                                   velocity=50.0, seed=n)


@pytest.mark.parametrize("precision", [DL_PLAIN_FP64, DL_MIXED])
@pytest.mark.parametrize("topology,n,per_strut,gauss,plastic", [
    ("bcc", 3, 1, 2, True),      # 216 elements: one block
    ("sc", 4, 1, 1, False),      # 300 elements, 125 nodes: several blocks of 32 elements
    ("bcc", 3, 2, 3, True),      # three points (the rolled loop)
    ("octet", 4, 2, 2, True),    # 12 slots at a node
    ("bcc", 14, 2, 2, True),     # 43,904 elements: one block per SM at its most threads (mixed), two (FP64)
    ("sc", 25, 3, 1, False),     # 152,100 elements, ragged: two blocks per SM
])
def test_same_bits_as_two_barriers(gpu, precision, topology, n, per_strut, gauss, plastic):
    spec = _spec(topology, n, per_strut, gauss, plastic)
    rng = np.random.default_rng(5)
    u = rng.normal(scale=1e-6, size=(spec.n_nodes, 3))
    th = rng.normal(scale=1e-3, size=(spec.n_nodes, 3))
    one, two = Lattice(spec, precision), Lattice(spec, precision)
    two.set_launch_shape(0, 128)
    watch = np.arange(0, spec.n_nodes, max(1, spec.n_nodes // 5))
    for g in (one, two):
        g.set_state(u=u, theta=th)
        g.set_sampling(4, watch, 20)
        for k in (7, 2, 31):   # odd and even runs: the slot sets start over with each launch
            g.run(k)
        g.synchronize()
    for a, b in zip(one.state(), two.state()):
        assert np.array_equal(a, b)
    (s1, r1, e1), (s2, r2, e2) = one.samples(), two.samples()
    assert np.array_equal(s1, s2) and np.array_equal(r1, r2)
    assert np.allclose(e1, e2, rtol=1e-12, atol=0)
    if plastic:
        for a, b in zip(one.history(), two.history()):
            assert np.array_equal(a, b)
    assert one.error_word() == two.error_word() == 0


def test_batch_of_small_lattices(gpu):
    specs = lattices.batch_lattices(n_lattices=5, seed=11, n_range=(2, 4))
    one, two = Batch(specs, DL_MIXED), Batch(specs, DL_MIXED)
    two.set_launch_shape(0, 64)
    for b in (one, two):
        b.run(60)
        b.synchronize()
    for k in range(len(specs)):
        for x, y in zip(one.lattice_state(k), two.lattice_state(k)):
            assert np.array_equal(x, y)
        e1, e2 = one.lattice_energies(k), two.lattice_energies(k)
        for key in ("kinetic", "potential", "dissipated"):
            assert e1[key] == pytest.approx(e2[key], rel=1e-12)


def test_barrier_failure_is_reported_and_cleared(gpu):
    """The split barrier of the one-barrier kernel gives up like the others."""
    spec = _spec("bcc", 4, 2, 2, True)
    g = Lattice(spec, DL_MIXED)
    g.set_barrier_test(2000, 1)
    g.run(4)
    assert g.error_word() & 0x4
    g.set_barrier_test(0, 0)
    g.clear_error()
    g.run(4)
    g.synchronize()


def test_models_of_different_sizes_side_by_side(gpu):
    """Each model's launches take their own shared memory, whatever was created
    after it."""
    big = Lattice(_spec("bcc", 12, 2, 2, False), DL_MIXED)
    ref = Lattice(_spec("bcc", 12, 2, 2, False), DL_MIXED)
    ref.run(10)
    ref.synchronize()
    small = Lattice(_spec("bcc", 4, 2, 2, False), DL_MIXED)
    for _ in range(5):
        small.run(2)
        big.run(2)
    small.synchronize()
    big.synchronize()
    for x, y in zip(big.state(), ref.state()):
        assert np.array_equal(x, y)
