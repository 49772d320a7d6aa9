"""Which passes a context runs is a matter of its own grid, solvent and
environment, not of the contexts made before it, and the tables they read are
made with the context."""
import ctypes

import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

from bgy3d_b200 import RismContext  # noqa: E402


def test_runtime_length_context_leaves_later_ones_alone(fixture_loader, monkeypatch):
    """A context made with the runtime-length passes (and timed: its schedule is
    kept for the shape) does not keep later ones of the shape on them."""
    meta, arr = fixture_loader("synth6_kh_n32")
    s = dict(meta["settings"])
    s.update({"closure": int(s["closure"]), "N": [36, 32, 54], "L": [4.5, 4.0, 6.75], "coarse-h": 0})
    monkeypatch.delenv("RISM3D_AUTOTUNE", raising=False)
    monkeypatch.setenv("RISM3D_GENERIC_PASSES", "1")
    a = RismContext(meta["solute"], meta["solvent"], s, arr["chi"])
    assert not a.tile_shapes()["f64"][3]
    monkeypatch.delenv("RISM3D_GENERIC_PASSES")
    b = RismContext(meta["solute"], meta["solvent"], s, arr["chi"])
    assert b.tile_shapes()["f64"][3] and b.tile_shapes()["f32"][3]
    a.close()
    b.close()


class Pool:
    """Bytes handed out by the device's default memory pool."""

    def __init__(self):
        self.rt = ctypes.CDLL("libcudart.so.12")
        self.h = ctypes.c_void_p()
        assert self.rt.cudaDeviceGetDefaultMemPool(ctypes.byref(self.h), 0) == 0

    def used(self):
        torch.cuda.synchronize()
        n = ctypes.c_uint64()
        assert self.rt.cudaMemPoolGetAttribute(self.h, 7, ctypes.byref(n)) == 0  # cudaMemPoolAttrUsedMemCurrent
        return n.value


@pytest.mark.parametrize("N", [(64, 64, 64), (54, 32, 108)])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_first_evaluation_makes_no_tables(fixture_loader, N, precision):
    """A first evaluation on a context, of a shape seen before, allocates nothing:
    the tables of the context's arithmetic are made with it."""
    meta, arr = fixture_loader("synth6_kh_n32")
    s = dict(meta["settings"])
    s.update({"closure": int(s["closure"]), "N": list(N), "L": [0.125 * n for n in N], "coarse-h": 0,
              "precision": precision})
    RismContext(meta["solute"], meta["solvent"], s, arr["chi"]).close()
    pool = Pool()
    for dt in (torch.float64,) if precision == "fp64" else (torch.float64, torch.float32):
        ctx = RismContext(meta["solute"], meta["solvent"], s, arr["chi"])
        T = torch.zeros(ctx.shape, device="cuda", dtype=dt)
        out = torch.empty_like(T)
        before = pool.used()
        assert before > 0
        ctx.jacobian_t1(T, T, out=out)
        ctx.iterate_t1(T, out=out)
        assert pool.used() <= before  # less: a context of an earlier test, collected meanwhile
        ctx.close()
