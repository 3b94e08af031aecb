"""The single-kernel step over the range of LJ types it promises (at most 64): its
table of type pairs stands in shared memory beside the phases' buffers, and from
34 types on the two pass the 48 KB a block has by default.  Types that are aliases
of the same few give the same trajectory bit for bit; 65 types step with the
separate kernels; and the autotuner, which times the single-kernel step among the
others, goes through at every count."""
import numpy as np
import pytest

import isspa_gb300 as ig

pytestmark = pytest.mark.gpu


def _aliased(s, big):
    nt = s.n_lj_types
    b = s.copy()
    alias = np.arange(big) % nt
    idx = np.asarray(s.nb_parm_index).reshape(nt, nt)
    b.n_lj_types = big
    b.nb_parm_index = idx[alias][:, alias].ravel().astype(np.int32)
    b.lj_ab = np.zeros((big * (big + 1) // 2, 2), np.float32)
    b.lj_ab[:len(s.lj_ab)] = s.lj_ab
    b.lj_type = (s.lj_type + nt * (np.arange(s.n_atoms) % (big // nt))).astype(np.int32)
    return b


@pytest.fixture(scope="module")
def system():
    return ig.synth.make_system(6, 22, 36.0, 5, seed=8, ff=ig.synth.forcefield(n_mc=5))


def _run(s, **o):
    eng = ig.Engine(s, field_split=4, **o)
    mode = eng.shapes()["integrator"]
    eng.step(9)
    out = eng.positions(), eng.velocities(), eng.device_status()
    eng.close()
    return mode, out


@pytest.mark.parametrize("types", [33, 34, 43, 44, 64, 65])
def test_single_kernel_step(system, types):
    ref = _run(system, integrator=2)[1]
    mode, got = _run(_aliased(system, types), integrator=3)
    assert mode == (3 if types <= 64 else 1)
    assert got[2] == 0
    assert np.array_equal(got[0], ref[0]) and np.array_equal(got[1], ref[1])


@pytest.mark.parametrize("types", [33, 34, 64, 65])
def test_autotune(system, types):
    eng = ig.Engine(_aliased(system, types))
    assert eng.autotune(reps=1)["integrator"] in (1, 2, 3)
    eng.step(2)
    assert eng.device_status() == 0
