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
