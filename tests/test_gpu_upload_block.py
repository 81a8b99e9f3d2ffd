"""Inputs that alternate about the size of a page-locked chunk (8 MiB): small ones are
packed into one device block, large ones copied array by array.  Either way the
results are the same, no allocation is made again, and contexts driven by several
threads copy side by side."""
import threading

import numpy as np
import pytest

import homs
from homs import _lib
from homs import workloads as W
from homs.model import BlochHighOrder

pytestmark = pytest.mark.gpu


def _run(obj, seq, st, mode, context=None):
    return homs.run_blocks(obj, seq, [(0, 12)], [False], BlochHighOrder("1111"), "f64", mode, st, context=context)


@pytest.mark.parametrize("mode", ["plain", "split"])
def test_alternating_sizes(gpu_context, mode):
    import torch
    cases = [W.high_order_workload(nspins=n, nsteps=12, ncoils=2) for n in (150_001, 60, 149_000, 131)]
    want = [_run(*c, mode) for c in cases]
    free = torch.cuda.mem_get_info()[0]
    for _ in range(3):
        for c, w in zip(cases, want):
            assert all(np.array_equal(a, b) for a, b in zip(_run(*c, mode), w))
        assert torch.cuda.mem_get_info()[0] == free


def test_contexts_of_several_threads(gpu_context):
    cases = [W.high_order_workload(nspins=n, nsteps=12, ncoils=2) for n in (400_001, 150_000, 300)]
    want = [_run(*c, "split") for c in cases]
    bad = []

    def work(k):
        ctx = _lib.Context()
        for i in range(6):
            c = (i + k) % len(cases)
            got = _run(*cases[c], "split", context=ctx)
            if not all(np.array_equal(a, b) for a, b in zip(got, want[c])):
                bad.append((k, i))
        ctx.close()

    threads = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad
