"""Pairs whose image direction is settled by one side (the other inside the box)
against the general form: a stretch of atoms moved just outside the upper face
makes the tiles that hold them take the general form, with the same geometry.
IS-SPA and nonbond forces against the oracle on those positions, and between the
field's splits and loops bit for bit per split."""
import numpy as np
import pytest

import isspa_gb300 as ig
import oracle as O
from parity import check_force

pytestmark = pytest.mark.gpu


def _system(out):
    s = ig.synth.make_system(15, 22, 40.0, 8, 4, ff=ig.synth.forcefield(n_mc=8))
    p = s.pos
    p[:, :3] = np.mod(p[:, :3], np.float32(s.box))
    if out:
        near = p[:, :3] < 4.0
        near[:100] = False  # (the first tiles keep the settled form)
        p[:, :3] = np.where(near, p[:, :3] + np.float32(s.box), p[:, :3])
        assert near.any()
    return s


@pytest.mark.parametrize("out", [False, True])
@pytest.mark.parametrize("split", [1, 2, 4, 8, 16])
def test_isspa_force(split, out):
    s = _system(out)
    o = O.Oracle(s)
    ref = o.isspa_force(o.mc_points(seed=s.seed, step=0))
    runs = []
    for vote in (2, 1):
        for apt in (1, 2):
            eng = ig.Engine(s, field_split=split, field_vote=vote, force_atoms_per_thread=apt, force_chunk=96)
            eng.zero_forces()
            eng.isspa_force()
            runs.append(eng.forces())
            assert eng.device_status() == 0
            eng.close()
    check_force(runs[0], ref, f"isspa split={split} out={out}")
    for f in runs[1:]:
        assert np.array_equal(f, runs[0])


@pytest.mark.parametrize("out", [False, True])
def test_nonbond_force(out):
    s = _system(out)
    eng = ig.Engine(s)
    eng.zero_forces()
    eng.nonbond_force()
    check_force(eng.forces(), O.Oracle(s).nonbond(7), f"nonbond out={out}")
    assert eng.device_status() == 0
