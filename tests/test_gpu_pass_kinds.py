"""The contexts whose z pass is not the radial one of up to three sites run the
specialised x and y passes: their results differ from the runtime-length ones'
by rounding (1e-10 of scale where the OZ solve may amplify it, else 1e-12 and, in
FP32, 2e-5: the bounds of the other comparisons between the families), and are
not the same to the last bit, which they would be if both ran one family."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

from bgy3d_b200 import RismContext, find_molecule  # noqa: E402

N, L = (54, 64, 108), (6.75, 8.0, 13.5)


def context(kind, meta, arr):
    s = dict(meta["settings"])
    s.update({"closure": int(s["closure"]), "N": list(N), "L": list(L), "coarse-h": 0})
    if kind == "pure":
        return RismContext(None, find_molecule("water"),
                           {"N": list(N), "L": 10.0, "rho": 0.033427745, "beta": 1.6889, "closure": "KH"}, None)
    if kind == "five sites":
        i = np.arange(5) % 3
        return RismContext(meta["solute"], [meta["solvent"][j] for j in i], dict(s, **{"no-renorm": True}),
                           np.ascontiguousarray(arr["chi"][np.ix_(i, i)]))
    rng = np.random.default_rng(41)  # chi - 1 on the k grid
    shape = (6, N[2], N[1], N[0] // 2 + 1)
    return RismContext(meta["solute"], meta["solvent"], s,
                       0.3 * (rng.standard_normal(shape) + 1j * rng.standard_normal(shape)))


@pytest.mark.parametrize("kind, cases", [("pure", [(torch.float64, 1e-10)]),
                                         ("five sites", [(torch.float64, 1e-12), (torch.float32, 2e-5)]),
                                         ("3D chi", [(torch.float64, 1e-12), (torch.float32, 2e-5)])])
def test_specialised_passes_of_every_kind(fixture_loader, kind, cases, monkeypatch):
    meta, arr = fixture_loader("synth6_kh_n32")
    monkeypatch.delenv("RISM3D_GENERIC_PASSES", raising=False)
    a = context(kind, meta, arr)
    monkeypatch.setenv("RISM3D_GENERIC_PASSES", "1")
    b = context(kind, meta, arr)
    g = torch.Generator(device="cuda").manual_seed(37)
    for dt, tol in cases:
        T = (torch.randn(a.shape, generator=g, device="cuda", dtype=torch.float64) * 0.1).to(dt)
        dT = (torch.randn(a.shape, generator=g, device="cuda", dtype=torch.float64) * 0.1).to(dt)
        for x, y in ((a.iterate_t1(T)[0], b.iterate_t1(T)[0]), (a.jacobian_t1(T, dT), b.jacobian_t1(T, dT))):
            scale = max(1.0, float(y.double().abs().max()))
            assert float((x.double() - y.double()).abs().max()) <= tol * scale, dt
            assert not torch.equal(x, y), dt
    a.close()
    b.close()
