"""Device vectors of the C calls that start off a 16-byte boundary: FP32 ones on
8 bytes (and the state of a Jacobian product and the preconditioner's vectors on
any element) give what aligned ones give, anything less is RISM3D_ERR_ARG.

They run other kernels of the same transforms, so they differ by rounding: 2e-5
of scale in FP32, 1e-12 in FP64, 1e-4 of max|z| for the preconditioner's 16 FP32
Krylov steps (the bounds of the other comparisons between those kernels)."""
import ctypes

import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

from bgy3d_b200 import RismContext, _abi  # noqa: E402


def shifted(x, k):
    """A copy of x that starts k elements off a 16-byte boundary."""
    y = torch.empty(x.numel() + k, dtype=x.dtype, device="cuda")[k:]
    y.copy_(x.flatten())
    return y


def ptr(x):
    return ctypes.c_void_p(x.data_ptr())


def close(got, want, tol):
    want = want.flatten().double()
    return float((got.double() - want).abs().max()) <= tol * max(1.0, float(want.abs().max()))


# old and new lengths, odd half rows, rows that are no multiple of eight values
@pytest.mark.parametrize("N", [54, 96, 108, 144])
def test_vectors_off_sixteen_bytes(fixture_loader, N):
    meta, arr = fixture_loader("synth6_kh_n32")
    s = dict(meta["settings"])
    s.update({"closure": int(s["closure"]), "N": N, "L": 0.125 * N})
    ctx = RismContext(meta["solute"], meta["solvent"], s, arr["chi"])
    assert ctx.coarse_grid() is not None
    L, h = _abi.lib(), ctx._h
    g = torch.Generator(device="cuda").manual_seed(29)
    T64 = torch.randn(ctx.shape, generator=g, device="cuda", dtype=torch.float64) * 0.1
    v64 = torch.randn(ctx.shape, generator=g, device="cuda", dtype=torch.float64) * 0.1
    T, v = T64.float(), v64.float()
    out, r = shifted(v, 2), (ctypes.c_double * 2)()

    assert L.rism3d_iterate_t1_f32(h, ptr(shifted(T, 2)), ptr(out), r) == _abi.OK
    F, norms = ctx.iterate_t1(T)
    assert close(out, F, 2e-5) and abs(r[0] - norms[0]) <= 2e-5 * max(1.0, norms[0])
    J = ctx.jacobian_t1(T, v)
    for x, dx, o in ((shifted(T, 1), v, torch.empty_like(v)), (shifted(T, 2), shifted(v, 2), out),
                     (T, shifted(v, 2), torch.empty_like(v)), (T, v, out)):
        o.fill_(float("nan"))
        assert L.rism3d_jacobian_t1_f32(h, ptr(x), ptr(dx), ptr(o)) == _abi.OK
        assert close(o.flatten(), J, 2e-5)
    o64 = torch.full_like(v64, float("nan"))
    assert L.rism3d_jacobian_t1(h, ptr(shifted(T64, 1)), ptr(v64), ptr(o64)) == _abi.OK
    assert close(o64.flatten(), ctx.jacobian_t1(T64, v64), 1e-12)

    z, z64 = ctx.precondition(T, v), ctx.precondition(T64, v64)
    for k in (1, 2):
        o = shifted(v, k)
        assert L.rism3d_precondition_f32(h, ptr(shifted(T, k)), ptr(shifted(v, k)), ptr(o)) == _abi.OK
        assert close(o, z, 1e-4)
    o = shifted(v64, 1)
    assert L.rism3d_precondition(h, ptr(shifted(T64, 1)), ptr(shifted(v64, 1)), ptr(o)) == _abi.OK
    assert close(o, z64, 1e-4)

    # less than a pair of values is refused, on the host
    assert L.rism3d_iterate_t1_f32(h, ptr(shifted(T, 1)), ptr(out), r) == _abi.ERR_ARG
    assert L.rism3d_jacobian_t1_f32(h, ptr(T), ptr(shifted(v, 1)), ptr(out)) == _abi.ERR_ARG
    assert L.rism3d_iterate_t1(h, ptr(shifted(T64, 1)), ptr(o64), r) == _abi.ERR_ARG
    assert L.rism3d_jacobian_t1(h, ptr(T64), ptr(v64), ptr(shifted(v64, 1))) == _abi.ERR_ARG
    ctx.close()
