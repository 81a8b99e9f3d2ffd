"""Packed transfers of small host arrays: a context of a few small calls page-locks
no memory (that takes longer than the calls), one that goes on gets its chunks, and
the results are the same bits before and after."""
import numpy as np
import pytest

import homs
from homs import workloads as W
from homs.model import BlochHighOrder

pytestmark = pytest.mark.gpu


def _resident_kb():
    """The process's resident memory, page-locked memory among it."""
    with open("/proc/self/status") as f:
        return next(int(line.split()[1]) for line in f if line.startswith("VmRSS"))


def _run(case, precision, mode, ctx):
    obj, seq, st = case
    return homs.run_blocks(obj, seq, [(0, 12)], [False], BlochHighOrder("1111"), precision, mode, st, context=ctx)


def test_few_small_calls_page_lock_nothing(homs_lib):
    case = W.high_order_workload(nspins=60, nsteps=12, ncoils=2)

    def calls(ctx):
        for precision, mode in (("f64", "plain"), ("f32", "split")):
            _run(case, precision, mode, ctx)
        homs.ResidentPhantom(case[0], "f64", "plain", context=ctx).close()

    with homs.Context(0) as ctx:
        calls(ctx)  # the library's own start
        before = _resident_kb()
        for _ in range(4):
            with homs.Context(0) as other:
                calls(other)
                assert _resident_kb() - before < 1024


@pytest.mark.parametrize("precision,mode", [("f64", "plain"), ("f32", "plain"), ("f32", "split")])
@pytest.mark.parametrize("nspins,calls", [(60, 20), (30_000, 150)])
def test_same_bits_on_either_side_of_the_chunks(homs_lib, precision, mode, nspins, calls):
    """60 spins pack into a chunk of 1 MB, 30,000 into one of 8 MB."""
    case = W.high_order_workload(nspins=nspins, nsteps=12, ncoils=2)
    with homs.Context(0) as ctx:
        want = _run(case, precision, mode, ctx)
        for _ in range(calls):
            assert all(np.array_equal(a, b) for a, b in zip(_run(case, precision, mode, ctx), want))
