"""Rules of the device sources that no run can show to be broken."""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "dynlattice_b200" / "csrc"


def _code(name):
    return re.sub(r"//.*", "", (CSRC / name).read_text())


def test_one_barrier_kernel_leaves_through_its_write_back():
    """A barrier wait that runs out ends the step loop; the block then writes its
    nodes' state back like after the last step."""
    body = _code("local.cuh")
    body = body[body.index("k_local("):]
    loop = body[body.index("for (int s = 0; s < c.nsteps"):]
    assert "return" not in re.sub(r"return reinterpret_cast", "", loop)
    assert re.search(r"if \(!grid_wait\([^;]*\)\) break;", loop)
    after = loop[loop.rindex("__syncthreads();"):]
    assert "st32(m.pos + n" in after and "st32(m.rot + n" in after and "m.vel[vel_ix(n, k)]" in after
    assert loop.count("st32(m.pos") == 1


def test_no_warp_collective_over_the_threads_that_happen_to_be_together():
    """__activemask() names the threads that run together just then, not those
    that take part in a collective."""
    for f in list(CSRC.glob("*.cuh")) + list(CSRC.glob("*.cu")):
        assert "__activemask" not in _code(f.name), f.name
