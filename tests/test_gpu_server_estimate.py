"""The server's admission estimate of a plain request covers the device memory that
the same run holds when it is prepared on its own (64 MB of the estimate are slack
for allocations' own overhead), and not several times as much."""
import numpy as np
import pytest

import homs
from homs import _lib
from homs import workloads as W
from homs.model import BlochHighOrder

pytestmark = pytest.mark.gpu


def _bytes(obj, seq, parts, exc, precision, ctx):
    """(estimate, device bytes of the prepared run after a run)."""
    params = {"sim_method": BlochHighOrder("1111"), "precision": precision, "homs_precision": "plain"}
    with homs.prepare_simulation(obj, seq, sim_params=params, parts=parts, excitation=exc, context=ctx) as plan:
        want = plan.run()
        held = plan.device_bytes()
    with homs.Server(slots=1) as srv:
        ticket = srv.submit(obj, seq, sim_params=params, parts=parts, excitation=exc)
        assert np.array_equal(srv.result(ticket), want)
        return srv.estimate(ticket), held


@pytest.mark.parametrize("precision", ["f32", "f64"])
@pytest.mark.parametrize("nspins,ncoils,nsteps,block", [
    (2_000_000, 1, 150, 150),  # 128 samples of phases per round, above the 384 MB of smaller phantoms
    (256, 32, 40_000, 40_000),  # partial sums in many parts of few spins
    (40_000, 8, 3_000, 1),  # a block per interval
    (40_000, 8, 3_000, 3_000)])
def test_estimate_covers_plain_runs(gpu_context, precision, nspins, ncoils, nsteps, block):
    obj, seq, _ = W.high_order_workload(nspins=nspins, nsteps=nsteps, ncoils=ncoils)
    parts, exc = homs.get_sim_ranges(seq, block)
    if precision == "f32":
        obj, seq = obj.astype(np.float32), seq.astype(np.float32)
    estimate, held = _bytes(obj, seq, parts, exc, precision, gpu_context)
    assert held <= estimate <= 3 * held + (128 << 20)


def test_unvalidated_requests_are_refused(gpu_context):
    """Sizes that no run accepts reach the estimate first: an error, not a crash."""
    import ctypes
    obj, seq, _ = W.high_order_workload(nspins=8, nsteps=4, ncoils=2)
    for precision in (_lib.HOMS_F32, _lib.HOMS_F64):
        for field, value in (("nspins", 0), ("nspins", -5), ("ncoils", 0), ("ncoils", -1), ("nnodes", 0), ("nblocks", 0)):
            keep = _lib._Keep()
            ph = _lib.host_phantom(obj, keep, precision)
            sq = _lib.host_sequence(seq, [(0, 4)], [False], keep, precision, homs.GAMMA)
            setattr(ph if hasattr(ph, field) else sq, field, value)
            opts = _lib.RunOptions(BlochHighOrder("1111").flags, _lib.HOMS_PLAIN)
            sig = np.zeros((4, 2), np.complex128)
            with homs.Server(slots=1) as srv:
                lib, ticket = _lib.load(), ctypes.c_int64()
                assert lib.homs_server_submit(srv.handle, ctypes.byref(ph), ctypes.byref(sq), ctypes.byref(opts), None,
                                              sig.ctypes.data, _lib.HOMS_HOST, ctypes.byref(ticket)) == 0
                assert lib.homs_server_wait(srv.handle, ticket.value, 60.0) == 1  # HOMS_EINVAL
