"""The block-per-cell list builder where it can go wrong: items of 8, 16 and 32
atoms, stencils past one staging pass, both of its tests, and the line to the
warp builder; the pair set (which a short list would lose pairs of) against
the FP64 oracle's."""
import numpy as np
import pytest

import systems as S

nbg = S.nbg
pytestmark = pytest.mark.gpu


def _lj(n, rho=0.8):
    u, v, L = nbg.workloads.lj_argon_lattice(n, rho=rho, seed=n, jitter=0.3)
    desc, keep = nbg.lennard_jones_descriptor(np.ones(n), L)
    return desc, keep, u


def _water(n_mol, R=0.9):
    sim = S.water_box(n_mol, seed=n_mol, R=R)
    desc, keep = nbg.system_descriptor(sim)
    return desc, keep, S.state(sim)[0]


# LJ cells are 2.8 wide: 27 cells from 549 atoms on, 343 from 6036; water
# cells of 1.0 nm hold ~105 atoms, so 27 of them take three passes; half cells
# (125 in the stencil) from ~900 molecules at R = 0.9 up where 16 atoms fill one
@pytest.mark.parametrize("case", ["lj-560", "lj-3000", "lj-6100", "lj-20000", "lj-sparse-5000", "water-950",
                                  "water-1200", "water-4096"])
def test_pair_set_of_cell_built_lists(gpu, oracle, case):
    kind, size = case.rsplit("-", 1)
    if kind == "lj":
        desc, keep, u = _lj(int(size))
    elif kind == "lj-sparse":
        desc, keep, u = _lj(int(size), rho=0.05)
    else:
        desc, keep, u = _water(int(size))
    which = nbg._abi.NBG_POT_EL if kind == "water" else nbg._abi.NBG_POT_LJ
    eng = nbg.Engine(desc, 0)
    assert eng.force_form() is not None  # on the list path
    np.testing.assert_array_equal(eng.pair_list(u, which), oracle.pair_list(desc, u, which))
    eng.close()
