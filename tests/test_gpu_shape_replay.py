"""Reported launch shapes are those that run, so that put back as options they
reproduce the engine: as created (where the voted field loop is a rule's choice, on
and off) and as tuned."""
import pytest

import isspa_gb300 as ig

pytestmark = pytest.mark.gpu


def _system(box):
    return ig.synth.make_system(20, 22, box, 5, seed=3, ff=ig.synth.forcefield(n_mc=5))


def _replay(s, shapes):
    keys = ("field_split", "force_chunk", "force_tail_chunk", "force_atoms_per_thread", "field_vote", "force_vote",
            "integrator", "field_tma")
    one_or_two = {k: 1 if shapes[k] else 2 for k in ("step_pdl", "isspa_fused", "force_overlap")}
    eng = ig.Engine(s, nonbond_chunk=shapes["nonbond_partners_per_item"], **{k: shapes[k] for k in keys}, **one_or_two)
    got = eng.shapes()
    eng.close()
    return got


@pytest.mark.parametrize("box, split, voted", [(60.0, 1, 1), (60.0, 4, 1), (60.0, 8, 0), (60.0, 16, 0), (90.0, 16, 1)])
def test_field_vote_as_created(box, split, voted):
    s = _system(box)  # (rmax 12 A: boxes of 5 and 7.5 rmax)
    eng = ig.Engine(s, field_split=split)
    shapes = eng.shapes()
    assert shapes["field_vote"] == voted
    assert _replay(s, shapes) == shapes
    plain = ig.Engine(s, field_split=split, field_vote=0).shapes()
    assert plain["field_vote"] == 0
    assert _replay(s, plain) == plain


def test_tuned_engine():
    s = _system(60.0)
    eng = ig.Engine(s)
    shapes = eng.autotune(reps=1)
    assert _replay(s, shapes) == shapes


@pytest.mark.parametrize("option, reported", [(0, 1), (1, 1), (2, 0)])
def test_merged_step_pdl(option, reported):
    """Merged steps launch as programmatic dependents unless told not to."""
    s = ig.synth.make_system(2, 22, 36.0, 5, seed=3, ff=ig.synth.forcefield(n_mc=5))
    shapes = ig.Engine(s, isspa_fused=1, field_split=8, integrator=1, step_pdl=option).shapes()
    assert shapes["step_pdl"] == reported
    assert _replay(s, shapes) == shapes


def test_tuned_merged_engine():
    s = ig.synth.make_system(2, 22, 36.0, 5, seed=3, ff=ig.synth.forcefield(n_mc=5))
    shapes = ig.Engine(s, integrator=1, isspa_fused=1).autotune(reps=1)
    assert shapes["isspa_fused"] == 1
    assert shapes["step_pdl"] == 1 or shapes["field_split"] == 4
    assert _replay(s, shapes) == shapes
