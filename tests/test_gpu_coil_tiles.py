"""The coil reduction's tiles (8-coil tiles, warps along the samples, spin
chunks) and copy widths: operands off the 16-byte boundary and odd leading
dimensions.  Bounds as in the reference's reduction test: 5e-13 (FP64) and 5e-6
(FP32) of sqrt(spins x samples x coils)."""
import ctypes
import math

import numpy as np
import pytest

from homs import _lib

pytestmark = pytest.mark.gpu


def _column_major(a, offset, ld):
    """Device copy of `a` (rows x cols) as columns of stride `ld`, `offset` real values past an aligned base."""
    import torch
    rows, cols = a.shape
    real = torch.float64 if a.dtype == np.complex128 else torch.float32
    buf = torch.full((offset + 2 * ld * cols,), float("nan"), dtype=real, device="cuda")
    v = buf[offset:].view(cols, 2 * ld)
    v[:, :2 * rows] = torch.as_tensor(np.ascontiguousarray(a.T).view(a.real.dtype), device="cuda")
    return buf, buf.data_ptr() + offset * buf.element_size()


@pytest.mark.parametrize("precision,offset,pad", [("f64", 0, 0), ("f64", 1, 1), ("f32", 0, 0), ("f32", 2, 1), ("f32", 1, 0)])
@pytest.mark.parametrize("nspins,nadc,nc", [(1, 16, 8), (31, 17, 9), (33, 32, 16), (64, 33, 17), (1000, 65, 33),
                                            (4099, 130, 65), (20001, 7, 1)])
def test_tiles_and_alignment(gpu_context, precision, offset, pad, nspins, nadc, nc):
    import torch
    rng = np.random.default_rng(11)
    ct = np.complex128 if precision == "f64" else np.complex64
    states, csm = ((rng.standard_normal((nspins, n)) + 1j * rng.standard_normal((nspins, n))).astype(ct)
                   for n in (nadc, nc))
    ld = nspins + pad
    keep_s, ps = _column_major(states, offset, ld)
    keep_c, pc = _column_major(csm, offset, ld)
    sig = torch.full((nc, nadc + 3), 7 - 3j, dtype=torch.complex128 if precision == "f64" else torch.complex64,
                     device="cuda")
    torch.cuda.synchronize()
    _lib.check(_lib.load().homs_coil_reduce(
        gpu_context.handle, _lib.HOMS_F64 if precision == "f64" else _lib.HOMS_F32, nspins, nadc, nc,
        ctypes.c_void_p(ps), ld, ctypes.c_void_p(pc), ld, ctypes.c_void_p(sig.data_ptr()), nadc + 3),
        gpu_context.handle)
    torch.cuda.synchronize()
    got = sig.cpu().numpy()
    ref = states.astype(np.complex128).T @ csm.astype(np.complex128)
    bound = 5e-13 if precision == "f64" else 5e-6
    assert np.linalg.norm(got[:, :nadc].T - ref) <= bound * math.sqrt(nspins * nadc * nc)
    assert np.all(got[:, nadc:] == 7 - 3j)


@pytest.mark.parametrize("precision", ["f64", "f32"])
@pytest.mark.parametrize("nspins,nadc,nc", [(63, 33, 9), (65, 33, 9), (8001, 64, 32), (37_888, 7, 3), (37_889, 7, 3),
                                            (75_776, 33, 17), (75_777, 33, 17), (60_000, 100, 3)])
def test_parts(gpu_context, precision, nspins, nadc, nc):
    """Both sides of the lines between parts of 256 spins (FP32 partial sums for FP32
    operands) and more parts with FP64 partial sums; the entry without allocation
    computes the same bits."""
    import torch
    rng = np.random.default_rng(12)
    ct = np.complex128 if precision == "f64" else np.complex64
    code = _lib.HOMS_F64 if precision == "f64" else _lib.HOMS_F32
    states, csm = ((rng.standard_normal((nspins, n)) + 1j * rng.standard_normal((nspins, n))).astype(ct)
                   for n in (nadc, nc))
    (ks, ps), (kc, pc) = _column_major(states, 0, nspins), _column_major(csm, 0, nspins)
    sig = [torch.zeros(nc, nadc, dtype=torch.complex128 if precision == "f64" else torch.complex64, device="cuda")
           for _ in range(2)]
    torch.cuda.synchronize()
    args = [(code, nspins, nadc, nc, ctypes.c_void_p(ps), nspins, ctypes.c_void_p(pc), nspins,
             ctypes.c_void_p(s.data_ptr()), nadc) for s in sig]
    _lib.check(_lib.load().homs_coil_reduce(gpu_context.handle, *args[0]), gpu_context.handle)
    _lib.check(_lib.load().homs_coil_reduce_noalloc(None, *args[1]), gpu_context.handle)
    torch.cuda.synchronize()
    got = sig[0].cpu().numpy()
    ref = states.astype(np.complex128).T @ csm.astype(np.complex128)
    bound = 5e-13 if precision == "f64" else 5e-6
    assert np.linalg.norm(got.T - ref) <= bound * math.sqrt(nspins * nadc * nc)
    assert np.array_equal(got, sig[1].cpu().numpy())
