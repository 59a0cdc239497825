"""Atoms lost under cubic boundaries (a coordinate that is not finite, or one so
many boxes out that its wrap means nothing) on the Verlet-list path: they are
listed by no atom, so the other accelerations are those of the system without
them, against a direct FP64 sum; in the small-system loop and in the list
builders' forms."""
import numpy as np
import pytest

import systems as S

nbg = S.nbg
pytestmark = pytest.mark.gpu

FORCE_TOL = 1e-5  # FP32 pair arithmetic, as everywhere


def _lj(u, L, pick, among, R=2.5):
    """Accelerations of the atoms `pick` by those of `among` (eps = sigma = m = 1), summed in FP64."""
    out = np.empty((len(pick), 3))
    for k, i in enumerate(pick):
        d = u[i] - u[among]
        d -= L * np.round(d / L)
        r2 = (d * d).sum(axis=1)
        d, r2 = d[(r2 < R * R) & (among != i)], r2[(r2 < R * R) & (among != i)]
        s6 = 1.0 / r2**3
        out[k] = (24.0 * (2.0 * s6 * s6 - s6) / r2) @ d
    return out


# n: the small-system loop; few cells (split test); cells of the hi test; the warp builder
@pytest.mark.parametrize("n", [700, 3000, 12000, 120000])
@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf, 1e25, -1e30])
def test_lost_atom_is_listed_by_nobody(gpu, n, value):
    rng = np.random.default_rng(n)
    u, v, L = nbg.workloads.lj_argon_lattice(n, seed=n, jitter=0.1)
    # among the first atoms and in the box's corner: where a lost atom would turn up
    lost = int(np.argmin((u * u).sum(axis=1)))
    w = u.copy()
    w[lost, rng.integers(3)] = value
    desc, keep = nbg.lennard_jones_descriptor(np.ones(n), L)
    eng = nbg.Engine(desc, 0)
    assert eng.force_form() is not None
    a = eng.accel(v.copy(), w)
    eng.close()
    rest = np.delete(np.arange(n), lost)
    assert not a[lost].any()
    # the atoms around the corner, and a sample of the others, without the lost one
    near = rest[np.argsort((u[rest] ** 2).sum(axis=1))[:40]]
    for pick in (near, rng.choice(rest, 40)):
        assert S.rel_rmse(a[pick], _lj(u, L, pick, rest)) <= FORCE_TOL
