"""The 1D solve shares its rows and radial points out over the host's threads;
chi, t and mu are those of one thread to the last bit."""
import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PROG = """
import os, sys
if sys.argv[1] == "1":
    os.sched_setaffinity(0, {min(os.sched_getaffinity(0))})
sys.path.insert(0, %r)
from bgy3d_b200 import find_molecule, rism_solvent
import hashlib
r = rism_solvent(find_molecule(sys.argv[2]), {"L": 10.0, "N": 64, "rho": 0.02, "beta": 1.6889, "closure": sys.argv[3],
                                              "rmax": 20.0, "nrad": int(sys.argv[4]), "norm-tol": 1e-10,
                                              "dielectric": float(sys.argv[5])})
print(hashlib.md5(r["susceptibility"].tobytes() + r["t"].tobytes()).hexdigest(), repr(r["free-energy"]))
"""


@pytest.mark.skipif(not hasattr(os, "sched_setaffinity"), reason="needs CPU affinity")
@pytest.mark.parametrize("mol, closure, nrad, eps", [("water, PR-SPC/E", "KH", 384, 78.4), ("hydrogen chloride", "PSE2", 288, 0.0),
                                                     ("Cl-, JC08, SPC/E", "KH", 128, 0.0)])
def test_result_does_not_depend_on_threads(mol, closure, nrad, eps):
    out = [subprocess.run([sys.executable, "-c", PROG % ROOT, one, mol, closure, str(nrad), str(eps)], check=True,
                          capture_output=True, text=True).stdout for one in ("1", "0")]
    assert out[0] == out[1] and out[0]
