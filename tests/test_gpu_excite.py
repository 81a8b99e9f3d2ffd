"""The excitation kernel of pulses without acquisition at the edges of its CTAs,
stages and unrolled steps, against the CPU oracle: FP64 at the engine's bar
1e-12 (130 rotations, each within a few 2^-53), FP32 at the reference's 3e-5.
"""
import numpy as np
import pytest

import homs
from conftest import nrmse
from homs import workloads as W
from homs.model import GAMMA, BlochHighOrder

pytestmark = pytest.mark.gpu

BAR = {"f64": 1e-12, "f32": 3e-5}


def _case(nspins, nsteps):
    obj, seq, st = W.high_order_workload(nspins=nspins, nsteps=nsteps, ncoils=2, rf=True)
    seq.adc[:] = False
    return obj, seq, st


def _check(oracle, obj, seq, st, parts, method, precision):
    exc = [True] * len(parts)
    ref = oracle.simulate_c(obj, seq, parts, exc, method.flags, st.xy, st.z)
    got = homs.run_blocks(obj, seq, parts, exc, method, precision, "plain", st)
    assert nrmse(got[1], ref[1]) <= BAR[precision] and nrmse(got[2], ref[2]) <= BAR[precision]


@pytest.mark.parametrize("precision", ["f64", "f32"])
@pytest.mark.parametrize("nspins,nsteps", [(1, 1), (31, 2), (63, 3), (64, 4), (65, 5), (128, 63), (129, 64), (33, 65),
                                           (70, 130)])
def test_edges(oracle, gpu_context, precision, nspins, nsteps):
    obj, seq, st = _case(nspins, nsteps)
    _check(oracle, obj, seq, st, [(0, nsteps)], BlochHighOrder("1111"), precision)


@pytest.mark.parametrize("precision", ["f64", "f32"])
def test_varying_steps_blocks_and_large_angles(oracle, gpu_context, precision):
    """Steps that change, blocks inside the pulse (frames of psi), no off-resonance
    term, fields from zero to several turns per step, infinite relaxation times."""
    obj, seq, st = _case(90, 70)
    rng = np.random.default_rng(3)
    seq.dt[:] = rng.uniform(1e-6, 6e-6, 70)
    seq.dt[10:20] = 2e-6
    seq.dt[60:70] = seq.dt[0] * (1 + 1e-12 * rng.standard_normal(10))
    seq.b1[20:30] = 0
    seq.gx[20:25] = seq.gy[20:25] = seq.gz[20:25] = seq.df[20:25] = 0
    seq.b1[40] = 0.02  # 2.6 turns in 3 us
    obj.T1[:5] = obj.T2[:5] = np.inf
    parts, _ = homs.get_sim_ranges(seq, 7, 7)
    for method in (BlochHighOrder("1111", True, True), BlochHighOrder("0000", False, True)):
        _check(oracle, obj, seq, st, parts, method, precision)


@pytest.mark.parametrize("turns", [0.0, 0.004, 0.028, 0.03, 0.1, 0.125, 0.13, 0.4, 3.0])
def test_half_angle_ranges(oracle, gpu_context, turns):
    """Half-angles on both sides of the lines between the two series and the general
    form (0.0281 and 0.1258 turns), within a warp and within the nodes of a step."""
    obj, seq, st = _case(70, 70)
    scale = turns / (GAMMA * float(seq.dt[0]) / 2)
    ramp = np.linspace(0.9, 1.1, 71)
    seq.b1[:] = scale * ramp * np.exp(1j * np.arange(71))
    seq.b1[33] = 0
    _check(oracle, obj, seq, st, [(0, 70)], BlochHighOrder("1111"), "f64")


@pytest.mark.parametrize("precision", ["f64", "f32"])
def test_zero_relaxation_times_and_nearly_equal_steps(oracle, gpu_context, precision):
    """Spins with T1 or T2 of zero (voxels outside the object) or far below the step
    relax at once, whatever the last bits of the steps: the factor is exp(-inf) = 0."""
    obj, seq, st = _case(90, 70)
    seq.dt[:] = seq.dt[0] * (1 + 1e-12 * np.random.default_rng(4).standard_normal(70))
    obj.T1[3:6] = obj.T2[5:9] = obj.T1[70:] = obj.T2[70:] = 0.0
    obj.T1[12] = obj.T2[13] = float(seq.dt[0]) / 800.0
    _check(oracle, obj, seq, st, [(0, 70)], BlochHighOrder("1111"), precision)
    parts, exc = [(0, 35), (35, 70)], [True, False]  # the samples that follow the pulse
    seq.adc[40:70:3] = True
    ref = oracle.simulate_c(obj, seq, parts, exc, BlochHighOrder("1111").flags, st.xy, st.z)
    got = homs.run_blocks(obj, seq, parts, exc, BlochHighOrder("1111"), precision, "plain", st)
    assert all(nrmse(g, r) <= BAR[precision] for g, r in zip(got, ref))
