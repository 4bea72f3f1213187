"""Rules of the device sources that no run can show to be broken."""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "dynlattice_b200" / "csrc"


def _code(name):
    return re.sub(r"//.*", "", (CSRC / name).read_text())


def test_one_barrier_kernel_writes_back_where_its_barrier_gives_up():
    """A block whose barrier wait runs out writes its nodes' state back, like after
    the last step, before it returns."""
    body = _code("local.cuh")
    body = body[body.index("k_local("):]
    loop = body[body.index("for (int s = 0; s < c.nsteps"):]
    give_up = loop[loop.index("if (!grid_wait("):]
    give_up = give_up[:give_up.index("return;")]
    for part in (give_up, loop[loop.index("if (last && own)"):]):
        assert "st32(m.pos + n" in part and "st32(m.rot + n" in part and "m.vel[vel_ix(n, k)]" in part
    assert loop.count("return;") == 1


def test_no_warp_collective_over_the_threads_that_happen_to_be_together():
    """__activemask() names the threads that run together just then, not those
    that take part in a collective."""
    for f in list(CSRC.glob("*.cuh")) + list(CSRC.glob("*.cu")):
        assert "__activemask" not in _code(f.name), f.name
