"""The threads of the 1D solve: the result of a solvent of several sites is that
of one thread to the last bit, and a host with other work on every core does not
hold a solve up.

A thread on a core that it shares with one busy process gets half of it, so even
a solve on one thread may take twice as long there; the bound is twice that."""
import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CORES = sorted(os.sched_getaffinity(0)) if hasattr(os, "sched_getaffinity") else []
PROG = """
import hashlib, os, sys, time
if sys.argv[1] == "1":
    os.sched_setaffinity(0, {min(os.sched_getaffinity(0))})
sys.path.insert(0, %r)
from bgy3d_b200 import RismError, find_molecule, rism_solvent
s = {"L": 10.0, "N": 64, "rho": 0.02, "beta": 1.6889, "closure": sys.argv[3], "rmax": 40.0, "nrad": int(sys.argv[4]),
     "norm-tol": 1e-10, "dielectric": 0.0}
w = find_molecule(sys.argv[2])
best = 1e9
for _ in range(int(sys.argv[5])):
    t0 = time.perf_counter()
    try:
        r = rism_solvent(w, s)
    except RismError as e:  # no convergence: alike on any number of threads
        print("error", e.code, 0.0)
        sys.exit()
    best = min(best, time.perf_counter() - t0)
print(hashlib.md5(r["susceptibility"].tobytes() + r["t"].tobytes()).hexdigest(), repr(r["free-energy"]), best)
""" % ROOT

pytestmark = pytest.mark.skipif(len(CORES) < 2, reason="needs two cores")


def solve(one, mol, closure, nrad, times=1):
    out = subprocess.run([sys.executable, "-c", PROG, "1" if one else "0", mol, closure, str(nrad), str(times)],
                         check=True, capture_output=True, text=True).stdout.split()
    return out[:-1], float(out[-1])


@pytest.mark.parametrize("mol, closure, nrad", [("water", "KH", 324), ("carbon disulfide", "HNC", 256),
                                                ("hydrogen chloride", "PSE3", 512)])
def test_several_sites_do_not_depend_on_threads(mol, closure, nrad):
    assert solve(True, mol, closure, nrad)[0] == solve(False, mol, closure, nrad)[0]


def test_busy_host_does_not_hold_a_solve_up():
    _, alone = solve(True, "water", "KH", 768, times=3)
    busy = [subprocess.Popen([sys.executable, "-c", "while True: pass"]) for _ in CORES]
    try:
        _, shared = solve(False, "water", "KH", 768, times=3)
    finally:
        for p in busy:
            p.kill()
            p.wait()
    assert shared < 4 * alone
