"""The adjoint at the sizes where its kernels change course, against the FP64
oracle: a window of two atoms, windows below and beyond one stage of the density
kernel (1024 atoms), more restrained atoms than one stage of the points kernel
(128), an atom in both restraint groups (weight zero), a window without a
restraint between restrained ones, point counts that end inside a block, and
fields on both sides of the Langevin branch (|E| = 5).  Tolerance 1e-5 of the
largest entry, as tests/test_gpu_adjoint.py: the fields and geometry are FP32."""
import numpy as np
import pytest

import isspa_gb300 as ig
import oracle as O

pytestmark = pytest.mark.gpu

TOL = 1e-5
N_MC = 3


def _window(chains, length, box, seed, groups=None, us=True):
    s = ig.synth.make_system(chains, length, box, N_MC, seed, ff=ig.synth.forcefield(n_mc=N_MC),
                             us=(10.0, 6.0) if us else None)
    if groups is not None:
        s.bias_list = np.array([(a, g) for g in (0, 1) for a in groups[g]], np.int32)
    return s


CASES = {
    "two atoms": lambda: [_window(2, 1, 30.0, 1)],
    "one stage exactly": lambda: [_window(64, 16, 60.0, 2)],
    "two stages, many restrained": lambda: [_window(75, 15, 62.0, 3, groups=(range(0, 150), range(300, 451)))],
    "batch": lambda: [_window(3, 11, 40.0, 4, groups=(range(0, 11), range(10, 22))), _window(4, 7, 40.0, 5, us=False),
                      _window(55, 20, 60.0, 6)],
}


@pytest.mark.parametrize("which", list(CASES))
def test_adjoint_sizes_match_oracle(which):
    wins = CASES[which]()
    eng = ig.Engine(wins)
    J, df, dg, dA, dB = eng.adjoint_mean_force([7])
    assert eng.device_status() == 0
    for w, s in enumerate(wins):
        got = (df[w], dg[w], dA[w], dB[w])
        if not s.us_on:
            assert J[w] == 0.0 and not any(np.any(g) for g in got)
            continue
        o = O.Oracle(s)
        pts = o.mc_points(seed=s.seed, step=7, window=w)
        assert abs(J[w] - o.mean_force(pts)) <= TOL * max(abs(J[w]), 1.0)
        for name, g, ref in zip(("dF", "dG", "dA", "dB"), got, o.adjoint(pts)[1:]):
            err = np.abs(g - ref).max() / max(np.abs(ref).max(), 1e-300)
            print(which, w, name, f"{err:.2e}")
            assert np.abs(g - ref).max() <= TOL * np.abs(ref).max(), (name, w)
