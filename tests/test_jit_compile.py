"""Runtime compilation of the step and adjoint kernels (no device needed): each
kernel is a program of its own, compiled beside the others and cached by itself."""
import json
import os
import subprocess
import sys
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent

SCRIPT = """
import ctypes as C, json, os, threading, time
from dynlattice_b200 import lattices
from dynlattice_b200.engine import load_library
lib = load_library()
d = lattices.lattice_impact(n=1).desc()
n, log = C.c_size_t(), C.create_string_buffer(1 << 16)
tasks = lambda: len(os.listdir("/proc/self/task"))
done, most = threading.Event(), [0]
def watch():
    while not done.wait(0.05):
        most[0] = max(most[0], tasks())
w = threading.Thread(target=watch)
w.start()
before, out = tasks(), []
for _ in range(2):
    wall = time.perf_counter()
    rc = lib.dl_jit_check(C.byref(d), int(os.environ["PREC"]), C.byref(n), log, C.c_size_t(1 << 16))
    out.append([rc, n.value, time.perf_counter() - wall, most[0] - before])
done.set()
w.join()
print(json.dumps(out))
"""


@pytest.mark.parametrize("precision", [0, 1])
def test_kernels_compile_side_by_side(tmp_path, precision):
    env = dict(os.environ, DL_JIT_CACHE=str(tmp_path), PREC=str(precision))
    r = subprocess.run([sys.executable, "-c", SCRIPT], cwd=ROOT, env=env, capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stderr[-2000:]
    first, second = json.loads(r.stdout.splitlines()[-1])
    assert first[0] == second[0] == 0 and first[1] == second[1] > 0
    # twelve step kernels and two adjoint kernels, each with its name
    for ext in (".cubin", ".names"):
        files = [p for p in tmp_path.iterdir() if p.suffix == ext]
        assert len([p for p in files if p.name.startswith("step_")]) == 12
        assert len([p for p in files if p.name.startswith("adjoint_")]) == 2
    assert first[3] >= min(len(os.sched_getaffinity(0)), 12) - 1   # threads beside the caller's
    assert second[2] < 0.2 * first[2]      # from the cache
