"""Which passes a context runs is a matter of its own grid, solvent and
environment, not of the contexts made before it."""
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
