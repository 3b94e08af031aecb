"""The merged step's bounded wait, made to run out from the host: a completion
count that its blocks cannot match.  The step reports ISSPA_ERR_TIMEOUT, neither
it nor the steps queued behind it (the rest of a graph of eight, further graphs)
integrate, and after the status reset the engine goes on from the unchanged state
with nothing of the failed steps' forces left."""
import numpy as np
import pytest

import isspa_gb300 as ig
from isspa_gb300 import abi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("graph", [True, False])
@pytest.mark.parametrize("split", [8, 16])
def test_no_step_integrates_after_a_timeout(split, graph):
    s = ig.synth.config_small(seed=1)
    make = lambda: ig.Engine(s, isspa_fused=1, field_split=split, integrator=1, use_graph=graph)
    eng, ref = make(), make()
    eng.step(3)
    ref.step(3)
    before = eng.positions(), eng.velocities()
    abi.check(abi.lib().isspa_debug_stall_barrier(eng._h), "stall")
    eng.step(17)
    assert eng.device_status() == abi.ERR_TIMEOUT
    assert np.array_equal(eng.positions(), before[0]) and np.array_equal(eng.velocities(), before[1])
    assert eng.get_step() == 3
    eng.step(8)  # still queued without a reset
    assert np.array_equal(eng.positions(), before[0]) and eng.get_step() == 3
    assert eng.device_status(reset=True) == abi.ERR_TIMEOUT
    assert eng.device_status() == 0
    assert not eng.forces().any()
    eng.step(17)
    ref.step(17)
    assert eng.device_status() == 0 and eng.get_step() == 20
    assert np.array_equal(eng.positions(), ref.positions()) and np.array_equal(eng.velocities(), ref.velocities())
