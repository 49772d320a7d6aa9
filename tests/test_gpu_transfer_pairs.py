"""The grid transfers by FFT along every axis at the pairs of lengths beyond
powers of two (odd half rows on either side, long axes): the preconditioner
with them equals the one with the dense transfer products
(RISM3D_DENSE_TRANSFERS=1) to the 1e-4 of max|z| of the other preconditioner
tests, in FP64 and FP32."""
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

from bgy3d_b200 import RismContext  # noqa: E402

# (fine points, half edges, coarse points)
CASES = [((162, 108, 64), (20.0, 13.0, 12.0), (54, 36, 32)), ((64, 162, 108), (12.0, 20.0, 20.0), (32, 54, 54)),
         ((108, 72, 162), (20.0, 12.0, 27.0), (54, 32, 72)), ((96, 96, 72), (12.0, 13.0, 13.0), (32, 36, 36)),
         ((324, 144, 96), (27.0, 18.0, 12.0), (72, 48, 32)), ((216, 288, 128), (20.0, 26.0, 20.0), (54, 72, 54)),
         ((288, 192, 64), (40.0, 36.0, 12.0), (108, 96, 32)), ((432, 64, 384), (36.0, 12.0, 40.0), (96, 32, 108)),
         ((486, 108, 64), (40.0, 18.0, 12.0), (108, 48, 32)), ((128, 486, 64), (20.0, 40.0, 12.0), (54, 108, 32))]


@pytest.mark.parametrize("N, L, nc", CASES)
def test_fft_transfer_pairs_match_dense(fixture_loader, N, L, nc, monkeypatch):
    meta, arr = fixture_loader("synth6_kh_n32")
    s = dict(meta["settings"])
    s.update({"closure": int(s["closure"]), "N": list(N), "L": list(L), "coarse-steps": 8})
    g = torch.Generator(device="cuda").manual_seed(31)
    out = {}
    for dense in ("0", "1"):
        monkeypatch.setenv("RISM3D_DENSE_TRANSFERS", dense)
        ctx = RismContext(meta["solute"], meta["solvent"], s, arr["chi"])
        assert ctx.coarse_grid() == nc
        if not out:
            T = torch.randn(ctx.shape, generator=g, device="cuda", dtype=torch.float64) * 0.3
            v = torch.randn(ctx.shape, generator=g, device="cuda", dtype=torch.float64)
        out[dense] = (ctx.precondition(T, v), ctx.precondition(T.float(), v.float()).double())
        ctx.close()
    scale = float(out["1"][0].abs().max())
    for z, ref in zip(out["0"], out["1"]):
        assert float((z - ref).abs().max()) < 1e-4 * scale
