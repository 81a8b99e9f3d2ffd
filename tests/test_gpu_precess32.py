"""The FP32 precession kernels (a walk over the nodes, then the signal in
parallel over samples) at the edges of their tiles and rounds.

Bounds: 3e-5, the reference's FP32 tolerance, against the FP64 oracle on the
short fixture; 2e-6 against an FP32 restatement of the reference's order of
operations, whose phases agree bit for bit, so that only sine, cosine, decay
and the products (each within 2 ulp of 6e-8, under 16 of them) differ.
"""
import numpy as np
import pytest

import homs
from conftest import nrmse
from homs import workloads as W
from homs.model import GAMMA, BlochHighOrder

pytestmark = pytest.mark.gpu

BAR = 3e-5


def _run(obj, seq, parts, exc, method, st, prec="f32"):
    return homs.run_blocks(obj, seq, parts, exc, method, prec, "plain", st)


@pytest.mark.parametrize("nspins,nsteps,ncoils", [
    (1, 1, 1), (3, 7, 2), (5, 8, 8), (31, 9, 9), (32, 63, 16), (33, 64, 17), (63, 65, 32), (64, 127, 33), (65, 128, 65),
    (130, 129, 8), (16384, 40, 3), (16385, 40, 3), (16415, 70, 1)])
def test_tile_edges(oracle, gpu_context, nspins, nsteps, ncoils):
    obj, seq, st = W.high_order_workload(nspins=nspins, nsteps=nsteps, ncoils=ncoils)
    method = BlochHighOrder("1111")
    ref = oracle.simulate_c(obj, seq, [(0, nsteps)], [False], method.flags, st.xy, st.z)
    got = _run(obj, seq, [(0, nsteps)], [False], method, st)
    assert all(nrmse(g, r) <= BAR for g, r in zip(got, ref))


@pytest.mark.parametrize("nspins", [70, 17000])
@pytest.mark.parametrize("mask,block", [("0000", 7), ("1010", 1), ("0101", 64), ("1111", 50)])
def test_sparse_samples_and_blocks(oracle, gpu_context, nspins, mask, block):
    """Every third node acquires; blocks restart the phase sum inside a stage and at its edges."""
    obj, seq, st = W.high_order_workload(nspins=nspins, nsteps=200, ncoils=5)
    seq.adc[:] = np.arange(201) % 3 == 2
    parts, exc = homs.get_sim_ranges(seq, block)
    method = BlochHighOrder(mask)
    ref = oracle.simulate_c(obj, seq, parts, exc, method.flags, st.xy, st.z)
    got = _run(obj, seq, parts, exc, method, st)
    assert all(nrmse(g, r) <= BAR for g, r in zip(got, ref))


def test_several_rounds(gpu_context):
    """More phases than one round's buffer holds: 120,000 spins x 2,000 samples in three rounds."""
    obj, seq, st = W.high_order_workload(nspins=120000, nsteps=2000, ncoils=2)
    method = BlochHighOrder("1111")
    want = _run(obj, seq, [(0, 2000)], [False], method, st, "f64")
    got = _run(obj, seq, [(0, 2000)], [False], method, st)
    assert all(nrmse(g, r) <= BAR for g, r in zip(got, want))


@pytest.mark.parametrize("nspins", [6, 17000])
def test_phase_sum_order(gpu_context, nspins):
    """The running sum over 9,000 nodes is rounded node by node in the reference's order."""
    w = W.config(1, spins_stride=41)
    seq = w.seq.view(0, 9003).astype(np.float32)
    seq.b1[:] = 0
    seq.adc[:] = False
    seq.adc[9000] = True
    n = min(nspins, len(w.obj))
    obj = w.obj[np.resize(np.arange(len(w.obj)), nspins)].astype(np.float32)
    f = np.float32
    st = homs.Mag(np.full(nspins, 1 - 0.5j, np.complex64), np.ones(nspins, f))
    method = BlochHighOrder("1111")
    got = _run(obj, seq, [(0, 9003)], [False], method, st)[1][:n]
    x, y, z = obj.x[:n], obj.y[:n], obj.z[:n]
    x2, y2, z2 = x * x, y * y, z * z
    r2 = (x2 + y2) + z2
    b = [x, x, y, z, x * y, z * y, f(3) * z2 - r2, x * z, x2 - y2, (f(3) * y) * x2 - (y2 * y), (x * z) * y,
         (f(5) * z2 - r2) * y, f(5) * (z2 * z) - (f(3) * z) * r2, (f(5) * z2 - r2) * x, x2 * z - y2 * z,
         (x2 * x) - (f(3) * x) * y2]
    dw = obj.dw[:n] / f(2 * np.pi * GAMMA)
    h = seq.h

    def field(k):
        b1 = (b[1] * h[1, k] + b[2] * h[2, k]) + b[3] * h[3, k]
        b2, b3 = b[4] * h[4, k], b[9] * h[9, k]
        for i in range(5, 9):
            b2 = b2 + b[i] * h[i, k]
        for i in range(10, 16):
            b3 = b3 + b[i] * h[i, k]
        return (((h[0, k] + b1) + b2) + b3) + dw

    acc, t, prev = np.zeros(n, f), f(0), field(0)
    for k in range(9003):
        nxt = field(k + 1)
        acc, t, prev = acc + (nxt + prev) * seq.dt[k], t + seq.dt[k], nxt
    phi = (f(-2 * np.pi * GAMMA) * (f(0.5) * acc)).astype(np.float64)
    want = (1 - 0.5j) * np.exp(-float(t) / obj.T2[:n].astype(np.float64)) * np.exp(1j * phi)
    assert np.max(np.abs(got - want) / np.abs(want)) <= 2e-6


def test_signal_does_not_depend_on_earlier_calls(homs_lib):
    """Five spins, the same call on one context after calls that leave small and large
    values where its padding spins' phases lie (partial sums of 256 coils): the same bits."""
    obj, seq, st = W.high_order_workload(nspins=5, nsteps=200, ncoils=8)
    other, oseq, ost = W.high_order_workload(nspins=5, nsteps=16, ncoils=256)
    method = BlochHighOrder("1111")
    with homs.Context(0) as ctx:
        def signal():
            return homs.run_blocks(obj, seq, [(0, 200)], [False], method, "f32", "plain", st, ctx)[0]

        signal()  # the workspace has its size
        found = []
        for scale in (0.0, 1.0, 1e5, 1e20):
            other.csm[:] = scale * np.exp(1j * np.arange(256))
            homs.run_blocks(other, oseq, [(0, 16)], [False], method, "f32", "plain", ost, ctx)
            found.append(signal())
    assert all(np.array_equal(f, found[0]) for f in found)


@pytest.mark.parametrize("nsteps,block", [(281, 1), (290, 2), (1100, 419), (1100, 400)])
def test_rounds_cut_at_blocks(gpu_context, nsteps, block):
    """120,000 spins: rounds of at most 69 blocks (the last of few nodes), a round whose
    samples (838) end with a block, and one that ends inside a later block."""
    obj, seq, st = W.high_order_workload(nspins=120000, nsteps=nsteps, ncoils=2)
    parts, exc = homs.get_sim_ranges(seq, block)
    method = BlochHighOrder("1111")
    want = _run(obj, seq, parts, exc, method, st, "f64")
    got = _run(obj, seq, parts, exc, method, st)
    assert all(nrmse(g, r) <= BAR for g, r in zip(got, want))
