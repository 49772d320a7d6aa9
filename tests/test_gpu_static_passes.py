"""The shape-specialised passes against the runtime-length ones on the same
inputs: every axis length that has them, 1 to 3 solvent sites, with and
without the renormalised long-range term, residual and Jacobian product.

The two families compute the same transforms with other splittings, so they
differ by rounding only: 1e-12 of scale in FP64, 2e-5 in FP32 (the tolerances
of the other comparisons between the families)."""
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

from bgy3d_b200 import RismContext  # noqa: E402

GRIDS = [(48, 64, 72), (72, 48, 64), (64, 72, 48), (96, 128, 144), (144, 96, 128), (128, 144, 96), (192, 256, 48),
         (48, 192, 256), (32, 36, 54), (54, 32, 36), (36, 54, 32), (54, 108, 162), (108, 162, 216), (162, 216, 108),
         (216, 288, 32), (288, 324, 36), (324, 32, 288), (384, 36, 324), (36, 384, 432), (432, 32, 486), (486, 432, 32),
         (32, 486, 384)]


def make(meta, arr, m, s, generic, monkeypatch):
    monkeypatch.setenv("RISM3D_AUTOTUNE", "0")
    if generic:
        monkeypatch.setenv("RISM3D_GENERIC_PASSES", "1")
    else:
        monkeypatch.delenv("RISM3D_GENERIC_PASSES", raising=False)
    return RismContext(meta["solute"], meta["solvent"][:m], s, arr["chi"][:m, :m].copy())


@pytest.mark.parametrize("m, norenorm", [(1, True), (2, False), (3, False), (3, True)])
@pytest.mark.parametrize("N", GRIDS)
def test_static_passes_match_runtime_length(fixture_loader, N, m, norenorm, monkeypatch):
    meta, arr = fixture_loader("synth6_kh_n32")
    s = dict(meta["settings"])
    # 0.25 A spacing keeps |k| inside the fixture's chi table
    s.update({"closure": int(s["closure"]), "N": list(N), "L": [0.125 * n for n in N], "coarse-h": 0,
              "no-renorm": norenorm})
    a = make(meta, arr, m, s, False, monkeypatch)
    b = make(meta, arr, m, s, True, monkeypatch)
    assert a.tile_shapes()["f64"][3] and a.tile_shapes()["f32"][3] and not b.tile_shapes()["f64"][3]
    g = torch.Generator(device="cuda").manual_seed(17)
    for dt, tol in ((torch.float64, 1e-12), (torch.float32, 2e-5)):
        T = (torch.randn(a.shape, generator=g, device="cuda", dtype=torch.float64) * 0.1).to(dt)
        dT = (torch.randn(a.shape, generator=g, device="cuda", dtype=torch.float64) * 0.1).to(dt)
        (Fa, na), (Fb, nb) = a.iterate_t1(T), b.iterate_t1(T)
        for x, y in ((Fa, Fb), (a.jacobian_t1(T, dT), b.jacobian_t1(T, dT))):
            scale = max(1.0, float(y.double().abs().max()))
            assert float((x.double() - y.double()).abs().max()) <= tol * scale, dt
        assert abs(na[0] - nb[0]) <= tol * max(1.0, nb[0]) and abs(na[1] - nb[1]) <= tol * max(1.0, nb[1])
    a.close()
    b.close()
