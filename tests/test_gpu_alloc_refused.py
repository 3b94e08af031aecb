"""Calls that allocate on first use, refused by the memory cap part way: the buffers
they did get do not make the next call take the others for present.  Under every
cap from the engine's own bytes up to what the call needs (32 bytes apart, so that
each buffer in turn is the first that does not fit) both calls are refused alike, and
with room for all of them they return what an uncapped engine returns."""
import numpy as np
import pytest

import isspa_gb300 as ig
from isspa_gb300 import abi

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def system():
    return ig.synth.make_system(2, 11, 34.0, 3, seed=8, ff=ig.synth.forcefield(n_mc=3), us=(10.0, 6.0))


def _engine(s, cap):
    try:
        return ig.Engine(s, mem_cap=cap)
    except ig.IsspaError as e:
        assert e.status == abi.ERR_NOMEM
        return None


def _smallest_cap(s):
    lo, hi = 4096, 1 << 30
    while hi - lo > 16:
        mid = (lo + hi) // 2
        eng = _engine(s, mid)
        if eng:
            eng.close()
            hi = mid
        else:
            lo = mid
    return hi


# (of the adjoint the value, summed in integers; its gradients' FP64 sums have no order)
CALLS = {"adjoint": lambda e: e.adjoint_mean_force([3])[:1], "point fields": lambda e: e.point_fields()}


@pytest.mark.parametrize("which", list(CALLS))
def test_refused_call_stays_refused(system, which):
    call = CALLS[which]
    cap = _smallest_cap(system)
    free = ig.Engine(system)
    ref = call(free)
    free.close()
    refused = 0
    for cap in range(cap, cap + (1 << 20), 32):
        eng = _engine(system, cap)
        got = []
        for _ in range(2):
            try:
                got.append(call(eng))
            except ig.IsspaError as e:
                assert e.status == abi.ERR_NOMEM
                got.append(None)
        assert (got[0] is None) == (got[1] is None)
        assert eng.device_status() == 0
        if got[0] is not None:
            for g in got:
                for a, b in zip(g, ref):
                    assert np.array_equal(a, b)
            break
        refused += 1
        eng.close()
    assert refused > 10 and got[0] is not None
