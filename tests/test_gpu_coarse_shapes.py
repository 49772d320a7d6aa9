"""The persistent coarse GMRES at every coarse grid of its plane form (32^3 to
96^3: whole basis, part of it and none of it resident in shared memory; odd
half rows at 54^3): equal to the graph-replayed
step-by-step kernels, and bitwise repeatable.

Both run 16 FP32 GMRES steps on the same operator with different roundings;
the bound is that of the other comparisons of the preconditioner (1e-4 of
max|z|)."""
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

from bgy3d_b200 import RismContext  # noqa: E402


@pytest.mark.parametrize("sites", [1, 3])
@pytest.mark.parametrize("n, L, nc", [(64, 12.0, 32), (72, 13.0, 36), (96, 18.0, 48), (108, 20.0, 54), (128, 24.0, 64), (144, 27.0, 72),
                                      (192, 36.0, 96)])
def test_persistent_shapes_match_graph(fixture_loader, n, L, nc, sites, monkeypatch):
    meta, arr = fixture_loader("synth6_kh_n32")
    s = dict(meta["settings"])
    s.update({"closure": int(s["closure"]), "N": n, "L": L, "coarse-steps": 16})
    g = torch.Generator(device="cuda").manual_seed(23)
    out = {}
    for mode in ("1", "0"):
        monkeypatch.setenv("RISM3D_COARSE_PERSIST", mode)
        ctx = RismContext(meta["solute"], meta["solvent"][:sites], s, arr["chi"][:sites, :sites].copy())
        assert ctx.coarse_grid() == (nc, nc, nc)
        if not out:
            T = torch.randn(ctx.shape, generator=g, device="cuda", dtype=torch.float64) * 0.3
            v = torch.randn(ctx.shape, generator=g, device="cuda", dtype=torch.float64)
        out[mode] = [ctx.precondition(T, v).clone() for _ in range(2)]
        assert ctx.coarse_driver() == ("persistent" if mode == "1" else "graph")
        ctx.close()
    assert torch.equal(out["1"][0], out["1"][1])
    scale = float(out["0"][0].abs().max())
    assert float((out["1"][0] - out["0"][0]).abs().max()) < 1e-4 * scale
