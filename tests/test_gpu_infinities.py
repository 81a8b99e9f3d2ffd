"""Infinite states and sensitivities: a component of the coil sums is infinite or
NaN exactly where the sum of its real products xr wr - xi wi, xr wi + xi wr is, and
the other samples and coils keep their values."""
import ctypes

import numpy as np
import pytest

import homs
from conftest import nrmse
from homs import _lib
from homs import workloads as W
from homs.model import BlochHighOrder

pytestmark = pytest.mark.gpu

INF = np.inf


def _same(got, ref, bar):
    g, r = (np.ascontiguousarray(v).view(v.real.dtype).astype(np.float64) for v in (got, ref))
    ok = np.isfinite(r)
    assert not ok.all() and ok.any()
    assert np.array_equal(g[~ok], r[~ok], equal_nan=True)
    assert nrmse(g[ok], r[ok]) <= bar


@pytest.mark.parametrize("precision,bar", [("f64", 1e-13), ("f32", 1e-6)])
@pytest.mark.parametrize("nspins,nadc,nc", [(3, 2, 3), (70, 33, 9), (3000, 20, 32)])
def test_coil_reduce(gpu_context, precision, bar, nspins, nadc, nc):
    import torch
    rng = np.random.default_rng(2)
    ct = np.complex128 if precision == "f64" else np.complex64
    x, w = ((rng.standard_normal((n, nspins)) + 1j * rng.standard_normal((n, nspins))).astype(ct) for n in (nadc, nc))
    w[0] = 1 + 1j
    x[1, nspins // 2] = complex(INF, 1)
    w[1, 0] = complex(-INF, 0)
    w[2, nspins - 1] = complex(1, INF)
    D = lambda a: torch.as_tensor(a, device="cuda")  # noqa: E731
    dx, dw, sig = D(x), D(w), torch.zeros(nc, nadc, dtype=torch.complex128 if precision == "f64" else torch.complex64,
                                          device="cuda")
    torch.cuda.synchronize()
    _lib.check(_lib.load().homs_coil_reduce(
        gpu_context.handle, _lib.HOMS_F64 if precision == "f64" else _lib.HOMS_F32, nspins, nadc, nc,
        ctypes.c_void_p(dx.data_ptr()), nspins, ctypes.c_void_p(dw.data_ptr()), nspins,
        ctypes.c_void_p(sig.data_ptr()), nadc), gpu_context.handle)
    torch.cuda.synchronize()
    xr, xi, wr, wi = (v.astype(np.float64) for v in (x.real, x.imag, w.real, w.imag))
    ref = np.empty((nc, nadc), np.complex128)
    with np.errstate(invalid="ignore"):
        for c in range(nc):
            ref[c].real = (xr * wr[c] - xi * wi[c]).sum(1)
            ref[c].imag = (xr * wi[c] + xi * wr[c]).sum(1)
    _same(sig.cpu().numpy(), ref, bar)


@pytest.mark.parametrize("precision,bar", [("f64", 1e-12), ("f32", 3e-5)])
@pytest.mark.parametrize("nspins,ncoils,nsteps", [(5, 3, 7), (90, 12, 40), (90, 20, 150)])
def test_precession(oracle, gpu_context, precision, bar, nspins, ncoils, nsteps):
    """Coils 1 and 2 have one infinite sensitivity each, then one spin an infinite state."""
    method = BlochHighOrder("1111")
    obj, seq, st = W.high_order_workload(nspins=nspins, nsteps=nsteps, ncoils=ncoils)
    obj.csm[0, 1] = complex(-INF, 0)
    obj.csm[nspins - 1, 2] = complex(1, INF)
    plan = [(0, nsteps)], [False], method.flags
    ref = oracle.simulate_c(obj, seq, *plan, st.xy, st.z)
    got = homs.run_blocks(obj, seq, *plan[:2], method, precision, "plain", st)
    _same(got[0], ref[0], bar)
    assert nrmse(got[1], ref[1]) <= bar and nrmse(got[2], ref[2]) <= bar
    obj, seq, st = W.high_order_workload(nspins=nspins, nsteps=nsteps, ncoils=ncoils)
    st.xy[1] = complex(INF, 1)
    ref = oracle.simulate_c(obj, seq, *plan, st.xy, st.z)
    got = homs.run_blocks(obj, seq, *plan[:2], method, precision, "plain", st)
    assert not np.isfinite(ref[0]).any() and np.isinf(np.ascontiguousarray(ref[0]).view(np.float64)).any()
    r, g = (np.ascontiguousarray(v).view(v.real.dtype).astype(np.float64) for v in (ref[0], got[0]))
    assert np.array_equal(g, r, equal_nan=True)
