"""Whole powers in expressions: what the evaluator and the set-up accept, and the
generated yield code against the expression's own tree."""
import copy
import ctypes as C
import subprocess
from pathlib import Path

import numpy as np
import pytest

import yield_cases as yc
from dynlattice_b200 import lattices
from dynlattice_b200.engine import load_library
from test_adjoint_cpu import NAMES, yield_source
from test_setup import inspect

ROOT = Path(__file__).resolve().parent.parent


def evaluate(expr, names=(), values=()):
    lib = load_library()
    n = (C.c_char_p * max(1, len(names)))(*[s.encode() for s in names])
    v = (C.c_double * max(1, len(values)))(*values)
    out = C.c_double()
    rc = lib.dl_eval_expression(expr.encode(), len(names), n, v, C.byref(out))
    return rc, out.value


@pytest.mark.parametrize("expr,x", [
    ("x^3 - 27", 3.0000000001),                       # cancels all but the last digits of the power
    ("x^5 - 2", 2.0 ** 0.2),
    ("x^4", 2.14061493270641e-78),                    # below the smallest normal number
    ("x^8", 1.453981324424731e-39),
    ("1/(x^7 - 2)", 2.0 ** (1.0 / 7.0) * (1 + 1e-12)),
    # as products, longer than a program may be
    pytest.param(" + ".join(f"(x + {k})^7" for k in range(200)), 0.3, id="200 powers"),
])
def test_expressions_with_powers_are_accepted(expr, x):
    rc, v = evaluate(expr, ["x"], [x])
    assert rc == 0, load_library().dl_last_error()
    assert v == pytest.approx(eval(expr.replace("^", "**")), rel=1e-13)


def test_long_yield_functions_are_accepted():
    """A yield program that is too long with its powers as products keeps pow."""
    spec = lattices.lattice_impact("bcc", n=1)
    spec.materials = [copy.copy(spec.materials[0])]
    terms = " + ".join(f"1e-9*(dx/1e3 + {k})^7" for k in range(150))
    spec.materials[0].yield_cond += f" + 0*({terms})"
    frames, _, mass, _ = inspect(spec)
    assert np.isfinite(frames).all() and (mass > 0).all()


@pytest.fixture(scope="module")
def policy(tmp_path_factory):
    d = tmp_path_factory.mktemp("yield")
    (d / "yield_policy.inc").write_text(yield_source(yc.material(0.5e-3), adjoint=False, host=False))
    so = d / "libyc.so"
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", f"-I{ROOT / 'dynlattice_b200' / 'csrc'}",
                    f"-I{d}", str(ROOT / "tests" / "cpp" / "yield_check.cpp"), "-o", str(so)], check=True,
                   capture_output=True)
    return C.CDLL(str(so))


def test_generated_yield_code_matches_the_expression(policy):
    """prep, f and grad as the step kernels call them.  Each value is a sum of
    at most 12 terms of at most 20 roundings: 1e-13 of the largest term."""
    rng = np.random.default_rng(2)
    dp = C.POINTER(C.c_double)
    for _ in range(200):
        r = rng.uniform(0.3e-3, 0.7e-3)
        area = np.pi * r * r
        cap = np.array([yc.SY / 3 ** 0.5 * area] * 2 + [yc.SY * area] + [yc.SY * 4 / 3 * r ** 3] * 2
                       + [yc.SY / 3 ** 0.5 * 2 / 3 * np.pi * r ** 3])
        args = np.concatenate([rng.uniform(-1.5, 1.5, 6) * cap, [rng.uniform(-1e3, 1e3)], [r, area]])
        f, g = C.c_double(), np.zeros(7)
        policy.yc_eval(args.ctypes.data_as(dp), C.byref(f), g.ctypes.data_as(dp))
        rc, want = evaluate(yc.COND, NAMES, args)
        assert rc == 0 and abs(f.value - want) < 1e-13 * 1.5 ** 8 * 12
        for k, d in enumerate(yc.DERIV):
            rc, want = evaluate(d, NAMES, args)
            scale = 8 * 1.5 ** 7 / (cap[k] if k < 6 else 1 / abs(want))
            assert rc == 0 and abs(g[k] - want) < 1e-13 * scale


def test_derivatives_of_the_case():
    """The case's own derivatives against central differences of its function."""
    r = 0.5e-3
    args = np.array([2e1, -3e1, -5e1, 1e-3, 2e-3, -1e-3, 10.0, r, np.pi * r * r])
    for k in range(7):
        h = max(abs(args[k]), 1e-3) * 1e-5
        up, dn = args.copy(), args.copy()
        up[k] += h
        dn[k] -= h
        fd = (evaluate(yc.COND, NAMES, up)[1] - evaluate(yc.COND, NAMES, dn)[1]) / (2 * h)
        assert evaluate(yc.DERIV[k], NAMES, args)[1] == pytest.approx(fd, rel=1e-4, abs=1e-9)
