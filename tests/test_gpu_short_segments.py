"""Short precession segments (few nodes, few samples) on the sequential kernel, on
both sides of the line that takes them there, against the CPU oracle.  Bounds as
for the parallel kernels: FP64 at the engine's bar 1e-12, FP32 at the reference's
3e-5."""
import ctypes

import numpy as np
import pytest

import homs
from conftest import nrmse
from homs import _lib
from homs import workloads as W
from homs.model import GAMMA, BlochHighOrder

pytestmark = pytest.mark.gpu

BAR = {"f64": 1e-12, "f32": 3e-5}


def _check(oracle, obj, seq, st, parts, exc, method, precision):
    ref = oracle.simulate_c(obj, seq, parts, exc, method.flags, st.xy, st.z)
    got = homs.run_blocks(obj, seq, parts, exc, method, precision, "plain", st)
    for g, r in zip(got, ref):
        assert g.shape == r.shape and (not r.size or nrmse(g, r) <= BAR[precision])


@pytest.mark.parametrize("precision", ["f64", "f32"])
@pytest.mark.parametrize("nspins,nsteps,ncoils,samples", [
    (1, 1, 1, 1), (255, 1, 2, 0), (256, 4, 1, 0), (257, 5, 1, 0), (300, 8, 3, 8), (70, 12, 33, 2), (70, 40, 2, 3),
    (520, 40, 3, 12), (16384, 9, 2, 9), (16385, 17, 2, 9), (16385, 31, 4, 20), (16385, 40, 4, 30), (100_001, 10, 2, 10),
    (100_001, 20, 3, 12)])
def test_tiles_and_lines(oracle, gpu_context, precision, nspins, nsteps, ncoils, samples):
    """Samples at the end of the segment: nodes, samples and coils on both sides of the lines."""
    obj, seq, st = W.high_order_workload(nspins=nspins, nsteps=nsteps, ncoils=ncoils)
    seq.adc[:] = np.arange(nsteps + 1) > nsteps - samples
    _check(oracle, obj, seq, st, [(0, nsteps)], [False], BlochHighOrder("1111"), precision)


@pytest.mark.parametrize("precision", ["f64", "f32"])
@pytest.mark.parametrize("mask,block", [("0000", 1), ("1010", 3), ("0101", 5), ("1111", 100)])
def test_among_pulses_and_long_segments(oracle, gpu_context, precision, mask, block):
    """Pulse, short segment, pulse, long segment, with blocks inside them; again from a prepared run."""
    obj, seq, st = W.high_order_workload(nspins=90, nsteps=160, ncoils=3, rf=True)
    exc = np.zeros(160, bool)
    exc[0:5] = exc[20:26] = exc[38:40] = True
    seq.excitation[:] = exc
    seq.adc[:] = np.arange(161) % 4 == 3
    seq.adc[:12] = False
    parts, flags = homs.get_sim_ranges(seq, block, 2)
    method = BlochHighOrder(mask)
    _check(oracle, obj, seq, st, parts, flags, method, precision)
    z0 = homs.Mag(np.zeros(90, complex), np.asarray(obj.rho).copy())
    ref = oracle.simulate_c(obj, seq, parts, flags, method.flags, z0.xy, z0.z)
    params = {"sim_method": method, "precision": precision}
    with homs.prepare_simulation(obj, seq, sim_params=params, parts=parts, excitation=flags, context=gpu_context) as plan:
        runs = [plan.run()[:, :, 0] for _ in range(4)]  # direct, captured, replayed
        state = plan.run(return_type="state")
    assert all(np.array_equal(r, runs[0]) for r in runs) and nrmse(runs[0], ref[0]) <= BAR[precision]
    assert nrmse(state.xy, ref[1]) <= BAR[precision] and nrmse(state.z, ref[2]) <= BAR[precision]


@pytest.mark.parametrize("precision", ["f64", "f32"])
def test_special_values(oracle, gpu_context, precision):
    """T1, T2 of zero and infinity, terms that the method leaves out, an infinite sensitivity."""
    obj, seq, st = W.high_order_workload(nspins=40, nsteps=8, ncoils=3)
    obj.T2[:4] = obj.T1[2:6] = np.inf
    obj.T2[7] = obj.T1[8] = 0.0
    method = BlochHighOrder("1100", True, False)
    want = oracle.simulate_c(obj, seq, [(0, 8)], [False], method.flags, st.xy, st.z)
    obj.dw[:] = np.nan
    seq.h[4:] = np.inf
    got = homs.run_blocks(obj, seq, [(0, 8)], [False], method, precision, "plain", st)
    assert all(nrmse(g, r) <= BAR[precision] for g, r in zip(got, want))
    obj.csm[0, 1] = complex(-np.inf, 0)
    want = oracle.simulate_c(obj, seq, [(0, 8)], [False], method.flags, st.xy, st.z)[0]
    got = homs.run_blocks(obj, seq, [(0, 8)], [False], method, precision, "plain", st)[0]
    assert np.array_equal(got[:, 1], want[:, 1].astype(got.dtype), equal_nan=True)
    assert nrmse(got[:, [0, 2]], want[:, [0, 2]]) <= BAR[precision]


@pytest.mark.parametrize("precision", ["f64", "f32"])
@pytest.mark.parametrize("nspins,ncoils,first,last", [(300, 2, 0, 1), (301, 3, 5, 25), (300, 33, 7, 16), (70, 2, 20, 160)])
def test_block_calls(oracle, gpu_context, precision, nspins, ncoils, first, last):
    """homs_precession_block on nodes first .. last of a longer sequence, on either
    kernel: the state one real past an aligned base, rows beyond the block's samples untouched."""
    import torch
    f, c = (np.float64, np.complex128) if precision == "f64" else (np.float32, np.complex64)
    dt = _lib.HOMS_F64 if precision == "f64" else _lib.HOMS_F32
    obj, seq, st = W.high_order_workload(nspins=nspins, nsteps=170, ncoils=ncoils)
    seq.adc[::5] = False
    n = int(seq.adc[first + 1:last + 1].sum())
    D = lambda a, t=f: torch.as_tensor(np.ascontiguousarray(np.asarray(a).astype(t)), device="cuda")  # noqa: E731
    keep = [D(v) for v in (obj.x, obj.y, obj.z, obj.rho, obj.T1, obj.T2, obj.dw)] + [D(obj.csm.T, c)]
    ph = _lib.Phantom(nspins, ncoils, dt, _lib.HOMS_DEVICE, *[k.data_ptr() for k in keep])
    node = [D(v) for v in (seq.t, seq.dt, seq.gx, seq.gy, seq.gz)] + [D(seq.b1, c), D(seq.df), D(seq.psi),
                                                                      D(seq.adc, np.uint8)]
    h = D(seq.h)
    hp = (ctypes.c_void_p * 16)(*[h[k].data_ptr() for k in range(16)])
    sq = _lib.Sequence(171, dt, _lib.HOMS_DEVICE, *[v.data_ptr() for v in node], hp, 0, None, None, None, GAMMA)
    raw = torch.zeros(2 * nspins + 1, dtype=keep[0].dtype, device="cuda")
    raw[1:] = torch.view_as_real(D(st.xy, c)).reshape(-1)
    z = D(st.z)
    state = _lib.State(raw.data_ptr() + raw.element_size(), z.data_ptr(), _lib.HOMS_DEVICE)
    sig = torch.zeros(ncoils, n + 3, dtype=keep[7].dtype, device="cuda")
    torch.cuda.synchronize()
    method = BlochHighOrder("1111")
    _lib.check(_lib.load().homs_precession_block(gpu_context.handle, ctypes.byref(ph), ctypes.byref(sq), first, last,
                                                 method.flags, ctypes.byref(state), sig.data_ptr(), n + 3),
               gpu_context.handle)
    torch.cuda.synchronize()
    ref = oracle.simulate_c(obj, seq, [(first, last)], [False], method.flags, st.xy, st.z)
    got = sig.cpu().numpy()
    assert nrmse(got[:, :n].T, ref[0]) <= BAR[precision] and np.all(got[:, n:] == 0)
    assert nrmse(raw[1:].cpu().numpy().view(c), ref[1]) <= BAR[precision] and float(raw[0]) == 0
    assert nrmse(z.cpu().numpy(), ref[2]) <= BAR[precision]


def test_full_size_readout_in_short_blocks(gpu_context):
    """350,000 spins x 2,000 samples x 32 coils: the parallel FP64 kernel and the split
    kernel, which both read the prefix table, against the sequential kernel, which does
    not: 500 block calls of 4 nodes, each from the state that the one before left."""
    import torch
    w = W.config(2)
    obj, seq, method = w.obj, w.seq, BlochHighOrder(w.mask)
    first = next(f for (f, l), rf in zip(w.parts, w.excitation) if not rf and seq.adc[f + 1:l + 1].sum() > 2000)
    first += int(np.flatnonzero(seq.adc[first + 1:])[0])
    last = first + 2000
    assert seq.adc[first + 1:last + 1].all()
    rng = np.random.default_rng(6)
    st = homs.Mag(obj.rho * np.exp(2j * np.pi * rng.uniform(size=len(obj))), 0.5 * obj.rho)
    D = lambda a, t=np.float64: torch.as_tensor(np.ascontiguousarray(np.asarray(a).astype(t)), device="cuda")  # noqa: E731
    keep = [D(v) for v in (obj.x, obj.y, obj.z, obj.rho, obj.T1, obj.T2, obj.dw)] + [D(obj.csm.T, np.complex128)]
    ph = _lib.Phantom(len(obj), obj.ncoils, _lib.HOMS_F64, _lib.HOMS_DEVICE, *[k.data_ptr() for k in keep])
    node = [D(v) for v in (seq.t, seq.dt, seq.gx, seq.gy, seq.gz)] + [
        D(seq.b1, np.complex128), D(seq.df), D(seq.psi), D(seq.adc, np.uint8)]
    h = D(seq.h)
    hp = (ctypes.c_void_p * 16)(*[h[k].data_ptr() for k in range(16)])
    sq = _lib.Sequence(len(seq.t), _lib.HOMS_F64, _lib.HOMS_DEVICE, *[v.data_ptr() for v in node], hp, 0, None, None, None,
                       GAMMA)
    xy, z = D(st.xy, np.complex128), D(st.z)
    state = _lib.State(xy.data_ptr(), z.data_ptr(), _lib.HOMS_DEVICE)
    sig = torch.zeros(obj.ncoils, 2000, dtype=torch.complex128, device="cuda")
    torch.cuda.synchronize()
    for k in range(0, 2000, 4):
        _lib.check(_lib.load().homs_precession_block(
            gpu_context.handle, ctypes.byref(ph), ctypes.byref(sq), first + k, first + k + 4, method.flags,
            ctypes.byref(state), sig[:, k:].data_ptr(), 2000), gpu_context.handle)
    torch.cuda.synchronize()
    want = sig.cpu().numpy().T, xy.cpu().numpy(), z.cpu().numpy()
    for mode, bars in (("plain", (1e-12, 1e-12, 1e-12)), ("split", (1e-6, 1e-12, 1e-12))):
        got = homs.run_blocks(obj, seq, [(first, last)], [False], method, "f64", mode, st)
        assert all(nrmse(g, r) <= bar for g, r, bar in zip(got, want, bars)), mode
