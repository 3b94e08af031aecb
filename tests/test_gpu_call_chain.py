"""The per-call force functions in a row, whose kernels depend programmatically on
the call's before them unless timed: the forces of untimed, timed and mixed
sequences agree bit for bit, over changing positions, in cutoff mode with list
builds, with restraints and with the fused launch."""
import numpy as np
import pytest

import isspa_gb300 as ig

pytestmark = pytest.mark.gpu

CALLS = ("bond_force", "angle_force", "dih_force", "isspa_force", "nonbond_force", "us_force")


@pytest.mark.parametrize("opts", [dict(), dict(isspa_fused=1, field_split=8), dict(nonbond_cutoff=9.0, nonbond_skin=0.5)])
def test_timed_and_untimed_calls_agree(opts):
    s = ig.synth.make_system(12, 22, 38.0, 8, 6, ff=ig.synth.forcefield(n_mc=8), us=(10.0, 8.0))
    eng = ig.Engine(s, **opts)
    rng = np.random.default_rng(1)
    pos = s.pos.copy()
    for k in range(12):
        pos[:, :3] += rng.normal(scale=0.1, size=(s.n_atoms, 3)).astype(np.float32)
        eng.set_positions(pos)
        got = []
        for timed in ([False] * 6, [True] * 6, [bool((k >> b) & 1) for b in range(4)] + [False, True]):
            eng.zero_forces()
            for name, t in zip(CALLS, timed):
                getattr(eng, name)(timed=t)
            got.append(eng.forces())
        assert np.array_equal(got[0], got[1]) and np.array_equal(got[0], got[2])
    assert eng.device_status() == 0
