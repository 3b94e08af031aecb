"""The nonbond pass at the edges of its tiles: 32 receiving atoms by groups of 32
partners, four groups in turn, stages of 128.  Single atoms, one atom below, at
and above a tile, a group and a stage; exclusion lists that cover whole groups
and cross stages; single terms; LJ tables too large for shared memory.  Against
the FP64 oracle with the suite's force tolerances (a pair's FP32 chain is about
ten roundings of 6e-8, times up to 14 through r^-13), and bit for bit between
partner stretches and between the two places of the LJ table."""
import numpy as np
import pytest

import isspa_gb300 as ig
import oracle as O
from parity import check_force

pytestmark = pytest.mark.gpu


def _system(chains, length, seed=3):
    box = max(34.0, (chains * length / 0.0051) ** (1 / 3))
    return ig.synth.make_system(chains, length, box, 5, seed, ff=ig.synth.forcefield(n_mc=5))


def _excluding(s, lists):
    """s with the exclusions of `lists` ({atom: later atoms}) in place of its own."""
    s = s.copy()
    cnt, flat = [], []
    for i in range(s.n_atoms):
        cnt.append(len(lists.get(i, ())))
        flat.extend(lists.get(i, ()))
    s.n_excl_cum = np.cumsum(cnt).astype(np.int32)
    s.excl_list = np.array(flat, np.int32)
    return s


def _nonbond(s, **opts):
    eng = ig.Engine(s, **opts)
    eng.zero_forces()
    eng.nonbond_force()
    f = eng.forces()
    assert eng.device_status() == 0
    eng.close()
    return f


@pytest.mark.parametrize("terms", [7, 3, 4])
@pytest.mark.parametrize("chains,length", [(2, 1), (1, 31), (4, 8), (3, 11), (1, 127), (8, 16), (3, 43), (1, 257)])
def test_tile_edges(chains, length, terms):
    s = _system(chains, length)
    f = _nonbond(s, nonbond_terms=terms)
    ref = O.Oracle(s).nonbond(terms)
    if ref.any():
        check_force(f, ref, f"nonbond {chains * length} atoms terms={terms}")
    else:  # (chains of one atom carry no charge)
        assert not f.any()
    for J in (128, 256, 1024):
        assert np.array_equal(_nonbond(s, nonbond_terms=terms, nonbond_chunk=J), f)


def test_single_atom():
    assert not _nonbond(_system(1, 1)).any()


@pytest.mark.parametrize("terms", [7, 5])
def test_long_exclusion_lists(terms):
    s = _excluding(_system(20, 15), {0: list(range(1, 300)), 5: list(range(32, 64)), 31: [32, 127, 128, 255, 256, 299],
                                     33: list(range(120, 140)), 130: list(range(131, 290)), 298: [299]})
    f = _nonbond(s, nonbond_terms=terms)
    check_force(f, O.Oracle(s).nonbond(terms), f"nonbond long exclusions terms={terms}")
    assert np.array_equal(_nonbond(s, nonbond_terms=terms, nonbond_chunk=1024), f)


@pytest.mark.parametrize("terms", [7, 1])
def test_large_lj_table(terms):
    """Types above 64 put the table in global memory: aliases of the same types
    give the same bits."""
    s = _system(7, 19)
    nt, big = s.n_lj_types, 70
    b = s.copy()
    alias = np.arange(big) % nt
    idx = np.asarray(s.nb_parm_index).reshape(nt, nt)
    b.n_lj_types = big
    b.nb_parm_index = idx[alias][:, alias].ravel().astype(np.int32)
    b.lj_ab = np.zeros((big * (big + 1) // 2, 2), np.float32)
    b.lj_ab[:len(s.lj_ab)] = s.lj_ab
    b.lj_type = (s.lj_type + nt * (np.arange(s.n_atoms) % (big // nt))).astype(np.int32)
    f = _nonbond(b, nonbond_terms=terms)
    check_force(f, O.Oracle(b).nonbond(terms), f"nonbond 70 LJ types terms={terms}")
    assert np.array_equal(f, _nonbond(s, nonbond_terms=terms))
