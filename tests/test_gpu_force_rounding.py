"""The accumulator's values as floats: the update converts the fixed-point force
of an atom on the device (two exact parts, or FP64 from 16384 on), the per-call
readback on the host in FP64.  Randomly placed atoms give forces on both sides
of the switch (some overlap, beyond what the status reports as overflow); every
one has to agree to the bit."""
import numpy as np
import pytest

import isspa_gb300 as ig

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("opts", [dict(isspa_terms=-1), dict(isspa_fused=1, field_split=16), dict(integrator=2)])
@pytest.mark.parametrize("seed", [1, 2])
def test_force_out_equals_host_conversion(opts, seed):
    s = ig.synth.make_system(12, 22, 36.0, 5, seed, ff=ig.synth.forcefield(n_mc=5))
    rng = np.random.default_rng(seed)
    s.pos[:, :3] = rng.uniform(0, 36.0, (s.n_atoms, 3)).astype(np.float32)
    a = ig.Engine(s, **opts)
    a.compute_forces()
    ref = a.forces()[:, :3]
    b = ig.Engine(s, **opts)
    out = [ig.host_array((s.n_atoms, 4)) for _ in range(3)]
    b.step_host(None, None, *out)
    big = np.abs(ref).max(axis=1)
    assert big.max() > 16384 and (big < 16384).any()
    assert np.array_equal(out[2][:, :3], ref)
