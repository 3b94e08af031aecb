"""The merged step (one launch per MD step for small engines with the fused
field + force launch) against the same engine's separate kernels, bit for bit:
the fused integrator (integrator 2) and the per-call sequence keep their own
kernels and run the same per-item code.  Cases: one window below and above a
nonbond stage of 128 partners and a stage per group of threads (44, 132, 300,
506 atoms), a restrained window with more than 128 restrained atoms, several
windows with and without restraints, terms switched off, and engines that keep
the branched step (too many atoms, cutoff mode)."""
import numpy as np
import pytest

import isspa_gb300 as ig
from isspa_gb300 import abi

pytestmark = pytest.mark.gpu

FF = {}


def _win(chains, length, seed, us=False, n_mc=5, box=None):
    ff = FF.setdefault(n_mc, ig.synth.forcefield(n_mc=n_mc))
    box = box or max(34.0, (chains * length / 0.0051) ** (1 / 3))
    return ig.synth.make_system(chains, length, box, n_mc, seed, ff=ff, us=(10.0, 8.0) if us else None)


def _many_restrained():
    s = _win(12, 25, 9, us=True)
    s.bias_list = np.array([(a, int(a >= 150)) for a in range(300)], np.int32)
    return s


CASES = {
    "44": (lambda: _win(2, 22, 1), {}),
    "132": (lambda: _win(6, 22, 2), {}),
    "300, 300 restrained": (_many_restrained, {}),
    "506": (lambda: _win(23, 22, 3), {}),
    "windows": (lambda: [_win(2, 22, 4, us=True), _win(7, 19, 5), _win(1, 1, 6), _win(3, 11, 7, us=True)], {}),
    "no nonbond": (lambda: _win(4, 22, 8), dict(nonbond_terms=abi.TERMS_NONE)),
    "nonbond LJ only": (lambda: _win(4, 22, 8), dict(nonbond_terms=1)),
    "too many atoms": (lambda: [_win(20, 22, 10), _win(20, 22, 11), _win(20, 22, 12)], {}),
    "cutoff": (lambda: _win(6, 22, 13), dict(nonbond_cutoff=12.0)),
}


@pytest.mark.parametrize("split", [4, 8, 16])
@pytest.mark.parametrize("which", list(CASES))
def test_merged_step_equals_separate_kernels(which, split):
    make, opts = CASES[which]
    s = make()
    runs = []
    for integ, pdl, graph in ((2, 2, True), (1, 1, True), (1, 2, True), (1, 1, False)):
        eng = ig.Engine(s, isspa_fused=1, field_split=split, integrator=integ, step_pdl=pdl, use_graph=graph, **opts)
        assert eng.shapes()["isspa_fused"] == 1
        eng.step(9)  # a graph of eight steps and one of one
        runs.append((eng.positions(), eng.velocities(), eng.us_com()[1], eng.get_step(), eng.device_status()))
        if integ == 1:  # the per-call sequence from here on agrees with the fused integrator's next step
            eng.compute_forces()
            eng.leapfrog()
        else:
            eng.step(1)
        runs[-1] += (eng.positions(),)
        eng.close()
    for r in runs:
        assert r[3] == 9 and r[4] == 0
        for a, b in zip(r, runs[0]):
            assert np.array_equal(a, b)
