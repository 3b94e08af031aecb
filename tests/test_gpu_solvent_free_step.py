"""The solvent-free step: nonbond and bonded terms in one launch, and in cutoff
mode the list check carried by the update.  Against the fused integrator, which
keeps the bonded terms and the check in launches of their own, bit for bit, over
graphs of eight steps and of one; restraints on a branch; terms switched off.
The list's rules on size: more cells than one block takes, more atoms than the
64-register pairs pass takes, rows longer than the entries fetched ahead."""
import numpy as np
import pytest

import isspa_gb300 as ig
from isspa_gb300 import abi

pytestmark = pytest.mark.gpu


def _win(chains, length, seed, us=False, box=None):
    box = box or max(34.0, (chains * length / 0.0051) ** (1 / 3))
    return ig.synth.make_system(chains, length, box, 5, seed, ff=ig.synth.forcefield(n_mc=5),
                                us=(10.0, 8.0) if us else None)


def _run(s, steps, **opts):
    eng = ig.Engine(s, isspa_terms=abi.TERMS_NONE, **opts)
    for n in steps:
        eng.step(n)
    out = (eng.positions(), eng.velocities(), eng.get_step(), eng.device_status())
    eng.close()
    assert out[3] == 0
    return out


CASES = {
    "31 atoms": (lambda: _win(1, 31, 1), {}),
    "windows": (lambda: [_win(2, 22, 2, us=True), _win(13, 19, 3), _win(1, 1, 4)], {}),
    "no nonbond": (lambda: _win(6, 22, 5), dict(nonbond_terms=abi.TERMS_NONE)),
    "LJ only": (lambda: _win(6, 22, 5), dict(nonbond_terms=1)),
    "no bonded terms": (lambda: _win(40, 1, 6), {}),
}


@pytest.mark.parametrize("cutoff", [0.0, 9.0])
@pytest.mark.parametrize("which", list(CASES))
def test_step_equals_fused_integrator(which, cutoff):
    make, opts = CASES[which]
    s = make()
    runs = [_run(s, (17, 1, 8), nonbond_cutoff=cutoff, **o, **opts)
            for o in (dict(integrator=2), dict(integrator=1), dict(integrator=1, step_pdl=2),
                      dict(integrator=1, use_graph=False))]
    for r in runs[1:]:
        assert r[2] == 26
        for k in (0, 1):
            assert np.array_equal(r[k], runs[0][k])


def test_list_rules_on_size():
    a, b = _win(400, 22, 7, box=120.0), _win(400, 22, 8, box=120.0)
    few = _run(a, (24,), nonbond_cutoff=3.0, nonbond_skin=4.0)  # 17^3 cells
    many = _run(a, (24,), nonbond_cutoff=3.0, nonbond_skin=0.5)  # 34^3 cells
    assert np.array_equal(many[0], few[0]) and np.array_equal(many[1], few[1])
    a.pnu = b.pnu = 0.0  # (collision draws belong to the window)
    single = [_run(s, (24,), nonbond_cutoff=9.0) for s in (a, b)]
    both = _run([a, b], (24,), nonbond_cutoff=9.0)  # 17600 atoms: the 40-register pass
    n = a.n_atoms
    for w, r in enumerate(single):
        assert np.array_equal(both[0][w * n:(w + 1) * n], r[0])
        assert np.array_equal(both[1][w * n:(w + 1) * n], r[1])


def test_rows_longer_than_fetched_ahead():
    s = _win(30, 22, 9)
    ref = _run(s, (10,), nonbond_cutoff=40.0, nonbond_skin=1.0)  # rows of several hundred
    got = _run(s, (10,), nonbond_cutoff=40.0, nonbond_skin=6.0)
    assert np.array_equal(ref[0], got[0]) and np.array_equal(ref[1], got[1])
