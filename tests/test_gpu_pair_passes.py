"""The shape-specialised x and y passes of contexts whose z pass is not the
radial one of up to three sites: the pure solvent (1 to 4 sites, 1 to 10 pair
fields, the molecular OZ step as a kernel between two z transforms) and a
solvent of five sites, against the runtime-length passes on the same inputs.

The families differ by rounding; the OZ solve (1 - rho W C)^-1 may amplify it,
so the pure solvent gets the 1e-10 of scale that it has against the oracle,
the others 1e-12 (FP64) and 2e-5 (FP32)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

from bgy3d_b200 import RismContext, find_molecule, hnc3d_run_solvent  # noqa: E402


def compare(make, monkeypatch, cases):
    monkeypatch.setenv("RISM3D_AUTOTUNE", "0")
    monkeypatch.delenv("RISM3D_GENERIC_PASSES", raising=False)
    a = make()
    monkeypatch.setenv("RISM3D_GENERIC_PASSES", "1")
    b = make()
    g = torch.Generator(device="cuda").manual_seed(23)
    for dt, tol in cases:
        T = (torch.randn(a.shape, generator=g, device="cuda", dtype=torch.float64) * 0.1).to(dt)
        dT = (torch.randn(a.shape, generator=g, device="cuda", dtype=torch.float64) * 0.1).to(dt)
        (Fa, na), (Fb, nb) = a.iterate_t1(T), b.iterate_t1(T)
        for x, y in ((Fa, Fb), (a.jacobian_t1(T, dT), b.jacobian_t1(T, dT))):
            scale = max(1.0, float(y.double().abs().max()))
            assert float((x.double() - y.double()).abs().max()) <= tol * scale, dt
        assert abs(na[0] - nb[0]) <= tol * max(1.0, nb[0]) and abs(na[1] - nb[1]) <= tol * max(1.0, nb[1])
    a.close()
    b.close()


@pytest.mark.parametrize("m, N", [(1, (32, 36, 48)), (2, (54, 32, 64)), (3, (96, 54, 32)), (3, (32, 32, 162)),
                                  (4, (36, 72, 54)), (4, (32, 64, 288)), (2, (32, 48, 486)), (3, (32, 512, 36))])
def test_pure_solvent(m, N, monkeypatch):
    w = find_molecule("water")
    sites = (w + [dict(w[1], x=[0.3, -0.8, 0.4])])[:m]
    s = {"N": list(N), "L": 10.0, "rho": 0.033427745, "beta": 1.6889, "closure": "KH"}
    compare(lambda: RismContext(None, sites, s, None), monkeypatch, [(torch.float64, 1e-10)])


@pytest.mark.parametrize("N", [(32, 36, 48), (54, 64, 108)])
def test_five_sites(fixture_loader, N, monkeypatch):
    meta, arr = fixture_loader("synth6_kh_n32")
    s = dict(meta["settings"])
    s.update({"closure": int(s["closure"]), "N": list(N), "L": [0.125 * n for n in N], "coarse-h": 0,
              "no-renorm": True})
    i = np.arange(5) % 3
    chi = np.ascontiguousarray(arr["chi"][np.ix_(i, i)])
    compare(lambda: RismContext(meta["solute"], [meta["solvent"][j] for j in i], s, chi), monkeypatch,
            [(torch.float64, 1e-12), (torch.float32, 2e-5)])


def test_solvent_energy_ignores_stale_device_memory():
    """The free energies after a context whose buffers were full of NaN is given back to the pool."""
    w = find_molecule("water")
    s = {"N": 48, "L": 10.0, "rho": 0.033427745, "beta": 1.6889, "norm-tol": 1e-12, "closure": "KH", "max-iter": 100}
    want = hnc3d_run_solvent(w, s)["free-energy"]
    for n in (48, 54, 64):
        ctx = RismContext(None, w, dict(s, N=n), None)
        ctx.jacobian_t1(torch.zeros(ctx.shape, device="cuda", dtype=torch.float64),
                        torch.full(ctx.shape, float("nan"), device="cuda", dtype=torch.float64))
        ctx.close()
        got = hnc3d_run_solvent(w, s)["free-energy"]
        assert abs(got - want) < 1e-8
