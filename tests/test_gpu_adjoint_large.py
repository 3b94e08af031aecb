"""The adjoint's own buffers on a system with many points: its force work list, over
the tiles that hold a restrained atom, stays within 2^20 items however many points
there are, and the longer chunks leave the value what the forces of the same step
give."""
import numpy as np
import pytest

import isspa_gb300 as ig

pytestmark = pytest.mark.gpu


def test_force_list_is_bounded():
    torch = pytest.importorskip("torch")
    n_mc = 3000
    s = ig.synth.make_system(200, 22, 95.0, n_mc, seed=3, ff=ig.synth.forcefield(n_mc=n_mc), us=(10.0, 5.0))
    atoms = np.arange(0, s.n_atoms, 100)  # one restrained atom per tile of 128 or more
    s.bias_list = np.stack([atoms, np.arange(len(atoms)) % 2], 1).astype(np.int32)
    eng = ig.Engine(s)
    eng.synchronize()
    before = torch.cuda.mem_get_info()[0]
    J = eng.adjoint_mean_force([0])[0][0]
    held = before - torch.cuda.mem_get_info()[0]
    points = 40 * eng.n_points  # raw fields and lambda
    assert held <= points + 16 * 2**20 + 8 * 2**20  # the list; everything small, allocation granularity
    # the same value from the step's forces: sum of +-n/2 F over the two groups
    eng.set_step(0)
    eng.zero_forces()
    for call in (eng.bond_force, eng.angle_force, eng.dih_force, eng.isspa_force, eng.nonbond_force):
        call()
    f = eng.forces().astype(np.float64)
    x = s.pos[:, :3].astype(np.float64)
    com = []
    for g in (0, 1):
        a = s.bias_list[s.bias_list[:, 1] == g, 0]
        m = s.raw_mass[a].astype(np.float64)
        com.append((m[:, None] * x[a]).sum(0) / m.sum())
    r = com[0] - com[1]
    r -= s.box * np.round(r / s.box)
    n = r / np.linalg.norm(r)
    sign = np.where(s.bias_list[:, 1] == 0, 0.5, -0.5)
    terms = sign * (f[s.bias_list[:, 0]] @ n)
    assert eng.device_status() == 0
    assert abs(J - terms.sum()) <= 1e-5 * np.abs(terms).sum()


def test_windows_of_very_different_sizes():
    """One restrained window beside a thousand of two atoms, half of them without a
    restraint: the large one gives what it gives alone, and only the restrained ones
    have a gradient."""
    n_mc = 20
    ff = ig.synth.forcefield(n_mc=n_mc)
    big = ig.synth.make_system(60, 22, 66.0, n_mc, seed=5, ff=ff, us=(10.0, 5.0))
    small = [ig.synth.make_system(2, 1, 30.0, n_mc, seed=6 + k, ff=ff, us=(10.0, 6.0) if k else None) for k in range(2)]
    wins = [big] + [small[k % 2] for k in range(1000)]
    eng = ig.Engine(wins, field_split=4)  # (the FP32 fields' order is the split's)
    got = eng.adjoint_mean_force([7])
    assert eng.device_status() == 0
    one = ig.Engine(big, field_split=4).adjoint_mean_force([7])
    for g, r in zip(got, one):  # FP64 sums in another order
        assert np.allclose(g[0], r[0], rtol=1e-12, atol=1e-12 * np.abs(r[0]).max())
    for w in (1, 2, 999, 1000):
        assert (got[0][w] != 0.0) == bool(wins[w].us_on)
        assert np.any(got[2][w]) == bool(wins[w].us_on)
