"""dJ/dT_g where the density product leaves FP32's range: every point lies inside rmax
of several atoms whose tabulated densities are far below (or above) one, so that the
products are 1e-40 and less (1e+40 and more) while each factor's share is what FP64
gives.  Tolerance 1e-5 of the largest entry, as tests/test_gpu_adjoint.py: the
geometry is FP32."""
import numpy as np
import pytest

import isspa_gb300 as ig
import oracle as O

pytestmark = pytest.mark.gpu

TOL = 1e-5
N_MC = 4


def _system(scale):
    s = ig.synth.make_system(2, 22, 25.0, N_MC, 3, ff=ig.synth.forcefield(n_mc=N_MC), us=(10.0, 6.0))
    s.g_table = (s.g_table * np.float32(scale)).astype(np.float32)
    # no zero in the core: a factor of its own, a tenth of the rest
    s.g_table[s.g_table == 0] = np.float32(0.1 * scale)
    return s


@pytest.mark.parametrize("scale", [1e-4, 1e-10, 1e-20, 1e3])
def test_density_gradient_range(scale):
    s = _system(scale)
    eng = ig.Engine(s)
    dg = eng.adjoint_mean_force([7])[2][0]
    o = O.Oracle(s)
    ref = o.adjoint(o.mc_points(seed=s.seed, step=7, window=0))[2]
    assert np.isfinite(ref).all() and np.abs(ref).max() > 0
    assert np.abs(dg - ref).max() <= TOL * np.abs(ref).max()


@pytest.mark.parametrize("small", [1e-12, 1e-20, 1e-30])
def test_few_small_factors(small):
    """Small only in the core, as a table exp(-u/kT) has it: shares of ordinary size
    for the core's bins beside shares that the core's factors make small; the bins are
    compared among those of their own size."""
    s = _system(1.0)
    core = np.arange(s.g_table.shape[1]) < 30
    s.g_table[:, core] = np.float32(small)
    dg = ig.Engine(s).adjoint_mean_force([7])[2][0]
    o = O.Oracle(s)
    ref = o.adjoint(o.mc_points(seed=s.seed, step=7, window=0))[2].reshape(s.g_table.shape)
    dg = dg.reshape(s.g_table.shape)
    assert np.abs(dg - ref).max() <= TOL * np.abs(ref).max()
    assert np.abs(ref[:, core]).max() > 0
    assert np.abs(dg - ref)[:, core].max() <= TOL * np.abs(ref[:, core]).max()
