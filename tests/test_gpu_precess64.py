"""The time-parallel FP64 precession kernel at the edges of its tiles (samples
per warp and CTA, 8-spin groups and 32-spin chunks, 8/16/32-coil tiles and
slices of 32 coils), against the CPU oracle.

The bound 1e-12 is the engine's FP64 bar: the fixture's phases stay below 100
rad, so their rounding (a few 2^-53 of the phase) is below 1e-13, and sums over
at most 100 spins add a few 2^-53 of the summands.
"""
import ctypes
import math

import numpy as np
import pytest

import homs
from conftest import nrmse
from homs import _lib
from homs import workloads as W
from homs.model import GAMMA, BlochHighOrder

pytestmark = pytest.mark.gpu

BAR = 1e-12


def _both(oracle, obj, seq, parts, exc, method, st):
    ref = oracle.simulate_c(obj, seq, parts, exc, method.flags, st.xy, st.z)
    return homs.run_blocks(obj, seq, parts, exc, method, "f64", "plain", st), ref


@pytest.mark.parametrize("nspins,nsteps,ncoils", [
    (1, 1, 1), (7, 15, 2), (8, 16, 8), (9, 17, 9), (31, 31, 16), (32, 32, 17), (33, 33, 32), (64, 63, 33),
    (65, 65, 65), (97, 127, 8), (40, 128, 9), (40, 129, 32), (33, 257, 1)])
def test_tile_edges(oracle, gpu_context, nspins, nsteps, ncoils):
    obj, seq, st = W.high_order_workload(nspins=nspins, nsteps=nsteps, ncoils=ncoils)
    got, ref = _both(oracle, obj, seq, [(0, nsteps)], [False], BlochHighOrder("1111"), st)
    assert all(nrmse(g, r) <= BAR for g, r in zip(got, ref))


@pytest.mark.parametrize("mask", ["0000", "1010", "0101", "1111"])
def test_sparse_samples_and_blocks(oracle, gpu_context, mask):
    """Every third node acquires, blocks of 7 intervals: the run is one segment."""
    obj, seq, st = W.high_order_workload(nspins=70, nsteps=200, ncoils=5)
    seq.adc[:] = np.arange(201) % 3 == 2
    parts, exc = homs.get_sim_ranges(seq, 7)
    got, ref = _both(oracle, obj, seq, parts, exc, BlochHighOrder(mask), st)
    assert all(nrmse(g, r) <= BAR for g, r in zip(got, ref))


def test_unused_terms_and_special_values(oracle, gpu_context):
    """A term that the method leaves out may hold anything; infinite T2 and a
    spin without transverse magnetisation are exact; T2 = 0 gives no signal."""
    obj, seq, st = W.high_order_workload(nspins=40, nsteps=40, ncoils=3)
    obj.T2[:4] = math.inf
    st.xy[5:9] = 0.0
    want = oracle.simulate_c(obj, seq, [(0, 40)], [False], BlochHighOrder("1100", True, False).flags, st.xy, st.z)
    obj.dw[:] = np.nan
    seq.h[4:] = np.inf
    got = homs.run_blocks(obj, seq, [(0, 40)], [False], BlochHighOrder("1100", True, False), "f64", "plain", st)
    assert all(nrmse(g, r) <= BAR for g, r in zip(got, want))
    assert np.all(got[1][5:9] == 0)
    obj.T2[:] = 0.0
    sig = homs.run_blocks(obj, seq, [(0, 40)], [False], BlochHighOrder("1100", True, False), "f64", "plain", st)[0]
    assert np.all(sig == 0)


@pytest.mark.parametrize("ncoils", [6, 20])
@pytest.mark.parametrize("low,high", [(0.05, 0.5), (0.5, 2.0), (2.0, 6.0), (5.0, 12.0), (12.0, 50.0), (0.01, 1e4)])
def test_decay_series(oracle, gpu_context, low, high, ncoils):
    """T2 about and on both sides of the lines between the decay series and 2^(t r2) (a
    tile's half span over T2 ln 2 equal to 1/16, and an eighth of that), also within
    one warp; both forms of the complex product."""
    obj, seq, st = W.high_order_workload(nspins=90, nsteps=300, ncoils=ncoils)
    seq.adc[:] = np.arange(301) % 2 == 0
    line = 16.0 * float(seq.t[128] - seq.t[0]) / math.log(2.0)
    obj.T2[:] = np.random.default_rng(5).permutation(np.geomspace(low, high, 90)) * line
    got, ref = _both(oracle, obj, seq, [(0, 300)], [False], BlochHighOrder("1111"), st)
    assert all(nrmse(g, r) <= BAR for g, r in zip(got, ref))


@pytest.mark.parametrize("sign", [1, -1])
def test_every_point_of_the_circle(oracle, gpu_context, sign):
    """Phases over all of the circle and up to 4e4 rad either way.  Bound: 300 roundings
    of the oracle's running sum at 4e4 rad, 300 * 4e4 * 2^-53 = 1.4e-9."""
    obj, seq, st = W.high_order_workload(nspins=200, nsteps=300, ncoils=3)
    obj.dw[:] = sign * np.linspace(0.0, 2e7, 200)
    got, ref = _both(oracle, obj, seq, [(0, 300)], [False], BlochHighOrder("1111"), st)
    assert all(nrmse(g, r) <= 1.4e-9 for g, r in zip(got, ref))


def test_block_call_with_state_off_16_bytes(oracle, gpu_context):
    """homs_precession_block accepts a state that is aligned to 8 bytes only."""
    import torch
    obj, seq, st = W.high_order_workload(nspins=45, nsteps=20, ncoils=4)
    D = lambda a: torch.as_tensor(np.ascontiguousarray(a), device="cuda")  # noqa: E731
    keep = [D(v) for v in (obj.x, obj.y, obj.z, obj.rho, obj.T1, obj.T2, obj.dw)] + [D(obj.csm.T)]
    ph = _lib.Phantom(45, 4, _lib.HOMS_F64, _lib.HOMS_DEVICE, *[k.data_ptr() for k in keep])
    node = [D(v) for v in (seq.t, seq.dt, seq.gx, seq.gy, seq.gz, seq.b1, seq.df, seq.psi, seq.adc.astype(np.uint8))]
    h = D(seq.h)
    hp = (ctypes.c_void_p * 16)(*[h[k].data_ptr() for k in range(16)])
    sq = _lib.Sequence(21, _lib.HOMS_F64, _lib.HOMS_DEVICE, *[v.data_ptr() for v in node], hp, 0, None, None, None,
                       GAMMA)
    raw = torch.zeros(2 * 45 + 1, dtype=torch.float64, device="cuda")
    raw[1:] = torch.view_as_real(D(st.xy)).reshape(-1)
    z = D(st.z)
    state = _lib.State(raw.data_ptr() + 8, z.data_ptr(), _lib.HOMS_DEVICE)
    sig = torch.zeros(4, 23, dtype=torch.complex128, device="cuda")
    torch.cuda.synchronize()
    method = BlochHighOrder("1111")
    _lib.check(_lib.load().homs_precession_block(gpu_context.handle, ctypes.byref(ph), ctypes.byref(sq), 0, 20,
                                                 method.flags, ctypes.byref(state), sig.data_ptr(), 23),
               gpu_context.handle)
    torch.cuda.synchronize()
    ref = oracle.simulate_c(obj, seq, [(0, 20)], [False], method.flags, st.xy, st.z)
    assert nrmse(sig.cpu().numpy()[:, :20].T, ref[0]) <= BAR
    assert nrmse(raw[1:].cpu().numpy().view(np.complex128), ref[1]) <= BAR
    assert nrmse(z.cpu().numpy(), ref[2]) <= BAR
    assert float(raw[0]) == 0.0 and torch.all(sig[:, 20:] == 0)


@pytest.mark.parametrize("block", [10**9, 100, 1])
def test_phase_of_long_runs_in_blocks(gpu_context, block):
    """10,000 nodes of a 30 mT/m readout, whole or cut into blocks, against extended
    precision.  The phase is a sum of 16 terms of at most 256 turns: some 22 roundings
    (products, kappas) of half an ulp of 2^-45 turns each, adding as their root sum of
    squares, 2 pi sqrt(22) 2^-46 = 4.2e-13 rad; a rounding running sum of kappa adds 5e-13."""
    ld, rng, ns, n = np.longdouble, np.random.default_rng(0), 60, 10000
    pos = rng.uniform(-0.1, 0.1, (3, ns))
    T2, dw = rng.uniform(0.03, 0.2, ns), rng.uniform(-2000.0, 2000.0, ns)
    csm = rng.standard_normal((ns, 3)) + 1j * rng.standard_normal((ns, 3))
    obj = homs.HO_Phantom(x=pos[0], y=pos[1], z=pos[2], rho=np.ones(ns), T1=10 * T2, T2=T2, dw=dw, csm=csm)
    dt = np.full(n, 1e-6)
    t = np.concatenate([[0.0], np.cumsum(dt)])
    h = np.zeros((16, n + 1))
    for k in (1, 2, 3):
        h[k] = 30e-3 * np.sin(2 * np.pi * (300 + 100 * k) * t + k)
    adc = np.arange(n + 1) > 0
    seq = homs.HO_DiscreteSequence(t, dt=dt, gx=h[1], gy=h[2], gz=h[3], b1=np.zeros(n + 1, complex), adc=adc,
                                   excitation=np.zeros(n, bool), h=h)
    parts, exc = homs.get_sim_ranges(seq, block)
    st = homs.Mag(np.full(ns, 0.6 + 0.3j), np.full(ns, 0.7))
    sig, xy, _ = homs.run_blocks(obj, seq, parts, exc, BlochHighOrder("1111"), "f64", "plain", st)
    two_pi = ld(2) * ld("3.14159265358979323846264338327950288")
    g = h[1:4].astype(ld)
    moment = np.cumsum(ld(0.5) * (g[:, :-1] + g[:, 1:]) * dt.astype(ld), axis=1)
    elapsed = np.cumsum(dt.astype(ld))[:, None]
    turns = -ld(GAMMA) * (moment.T @ pos.astype(ld)) - elapsed * (dw.astype(ld) / two_pi)
    phase, e = two_pi * (turns - np.rint(turns)), np.exp(-elapsed / T2.astype(ld))
    re = e * (ld(0.6) * np.cos(phase) - ld(0.3) * np.sin(phase))
    im = e * (ld(0.6) * np.sin(phase) + ld(0.3) * np.cos(phase))
    cr, ci = csm.real.astype(ld), csm.imag.astype(ld)
    for got, want in ((sig, ((re @ cr - im @ ci), (re @ ci + im @ cr))), (xy, (re[-1], im[-1]))):
        d = (got.real - want[0]) ** 2 + (got.imag - want[1]) ** 2
        assert float(np.sqrt(d.sum() / (want[0] ** 2 + want[1] ** 2).sum())) <= 4.2e-13
