"""A yield function with whole powers up to 8, a branch and divisions by section
values on the GPU: the compiled kernels and the interpreted program against the
oracle, which evaluates the expression as it stands."""
import numpy as np
import pytest

import yield_cases as yc
from dynlattice_b200 import lattices
from dynlattice_b200.abi import DL_MIXED, DL_PLAIN_FP64
from dynlattice_b200.engine import Lattice
from helpers import rel_err
from oracle_ffi import Oracle

pytestmark = pytest.mark.gpu


# the tolerances of the other elastoplastic runs against the oracle
@pytest.mark.parametrize("precision,tol", [(DL_PLAIN_FP64, 1e-9), (DL_MIXED, 1e-5)])
@pytest.mark.parametrize("interpreted", [False, True])
def test_yield_with_powers_matches_oracle(gpu, monkeypatch, precision, tol, interpreted):
    spec = lattices.lattice_impact("bcc", n=2, velocity=20.0, dt=5e-8, radius_jitter=0.0)
    spec.materials = [yc.material(spec.materials[0].radius)]
    if interpreted:
        monkeypatch.setenv("DL_NO_JIT", "1")
    g = Lattice(spec, precision)
    assert g.info()["jit"] == (not interpreted)
    assert g.launch_shape(400)["kernel"] == "one_barrier"
    o = Oracle(spec, threads=4)
    o.run(400)
    g.run(399)
    g.run(1)
    g.synchronize()
    assert rel_err(g.state()[0], o.state()[0]) < tol
    assert g.energies()["dissipated"] > 0
    assert g.energies()["dissipated"] == pytest.approx(o.energies()["dissipated"], rel=max(tol, 1e-9) * 100)
