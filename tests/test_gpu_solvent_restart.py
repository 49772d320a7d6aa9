"""A pure-solvent solve restarted from its own fixed point is over before the
pages of its result buffers have all been touched.  What it returns is the same
to the last bit whether those pages are fresh (mapped while the device works,
chi - 1 alone 102 MB here) or were there before the call."""
import ctypes

import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

from bgy3d_b200 import _abi, find_molecule, hnc3d_run_solvent  # noqa: E402
from bgy3d_b200.solver import _dptr, _sites, problem_data  # noqa: E402


def test_restart_at_the_fixed_point_is_bitwise():
    w = find_molecule("water")
    s = {"N": 128, "L": 12.0, "rho": 0.033427745, "beta": 1.6889, "closure": "KH", "norm-tol": 1e-10, "max-iter": 100}
    t = hnc3d_run_solvent(w, s)["RESTART"]
    # the same call into buffers whose pages exist
    pd = problem_data(s)
    chi = np.full((6, 128, 128, 65), complex(1.5, 1.5))
    t_out, g = np.full(t.shape, 1.5), np.full(t.shape, 1.5)
    res = _abi.SolventResult()
    rc = _abi.lib().rism3d_solvent_solve(ctypes.byref(pd), 3, _sites(w), _dptr(t), _dptr(t_out), _dptr(chi), _dptr(g),
                                         ctypes.byref(res))
    assert rc == _abi.OK and res.newton_iters == 0
    assert np.array_equal(t_out, t)
    for _ in range(6):
        r = hnc3d_run_solvent(w, s, restart=t)
        assert np.array_equal(r["RESTART"], t)
        assert np.array_equal(r["GVV"], g)
        assert np.array_equal(r["susceptibility-3d"], chi)
