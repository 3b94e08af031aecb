"""isspa_step_host with mapped buffers on a step that gives up: the buffers hold the
state that the engine holds, unchanged, as copies after the step would."""
import numpy as np
import pytest

import isspa_gb300 as ig
from isspa_gb300 import abi

pytestmark = pytest.mark.gpu

STEPS = {"merged": dict(integrator=1, isspa_fused=1, field_split=8), "fused integrator": dict(integrator=2),
         "single kernel": dict(integrator=3)}


@pytest.mark.parametrize("graph", [True, False])
@pytest.mark.parametrize("which", list(STEPS))
def test_buffers_hold_the_unchanged_state(which, graph):
    s = ig.synth.make_system(6, 22, 36.0, 5, seed=8, ff=ig.synth.forcefield(n_mc=5))
    eng = ig.Engine(s, use_graph=graph, **STEPS[which])
    n = eng.n_atoms
    pin, vin, pout, vout, fout = (ig.host_array((n, 4)) for _ in range(5))
    eng.step_host(None, None, None, None, fout)
    force = fout.copy()
    pin[:], vin[:] = eng.positions(), eng.velocities()
    vin[:, :3] *= 0.5
    for a in (pout, vout, fout):
        a[:] = -7.0
    abi.check(abi.lib().isspa_debug_stall_barrier(eng._h), "stall")
    eng.step_host(pin, vin, pout, vout, fout)
    assert eng.device_status(reset=True) == abi.ERR_TIMEOUT
    assert np.array_equal(pout, pin) and np.array_equal(vout, vin) and np.array_equal(fout, force)
    assert np.array_equal(eng.positions(), pin) and np.array_equal(eng.velocities(), vin)
