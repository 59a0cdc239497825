"""Energies of states with a lost atom. A NaN coordinate of either sign counts
as beyond every cutoff (no comparison with it holds), in both energy kernels; a
position past the minimum-image loop's cap is refused wherever a listed pair
reaches it, beyond the cutoff too."""
import numpy as np
import pytest

import systems as S

nbg = S.nbg
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("system", ["pairs", "list-split", "list-hi"])
def test_nan_position_of_either_sign(gpu, system):
    n = {"pairs": 300, "list-split": 3000, "list-hi": 12000}[system]
    u, v, L = nbg.workloads.lj_argon_lattice(n, seed=n, jitter=0.1)
    desc, keep = nbg.lennard_jones_descriptor(np.ones(n), L)
    if system == "pairs":
        desc.flags |= nbg._abi.NBG_FLAG_ALL_PAIRS
    eng = nbg.Engine(desc, 0)
    whole = eng.energy(u, v)
    got = []
    for value in (np.nan, -np.nan):
        w = u.copy()
        w[17, 1] = value
        got.append(eng.energy(w, v))
    eng.close()
    assert got[0] == got[1]
    d = u[17] - np.delete(u, 17, axis=0)
    d -= L * np.round(d / L)
    r2 = (d * d).sum(axis=1)
    s6 = (1.0 / np.minimum(r2, 2.5**2)) ** 3  # the atom's pairs, and the same at the cutoff
    cut = 2.5**-6
    lost = 4.0 * ((s6 * s6 - s6).sum() - (n - 1) * (cut * cut - cut))
    assert abs(got[0]["lennard_jones"] - (whole["lennard_jones"] - lost)) <= 1e-11 * abs(whole["lennard_jones"])


# a simple cubic lattice of spacing 2.6: every listed pair (radius 2.8) is
# beyond the cutoff, 2.5, and no pair's arithmetic is reached; and a liquid
@pytest.mark.parametrize("boxes", [70000, 2**33])
@pytest.mark.parametrize("system,n", [("lattice", 12**3), ("lattice", 20**3), ("liquid", 3000), ("liquid", 12000)])
def test_position_past_the_image_cap_is_refused(gpu, system, n, boxes):
    if system == "lattice":
        side = round(n ** (1 / 3))
        g, L = 2.6 * np.arange(side) + 0.3, 2.6 * side
        u = np.stack(np.meshgrid(g, g, g, indexing="ij"), -1).reshape(-1, 3)
        v = np.ones_like(u)
    else:
        u, v, L = nbg.workloads.lj_argon_lattice(n, seed=n, jitter=0.1)
    desc, keep = nbg.lennard_jones_descriptor(np.ones(n), L)
    eng = nbg.Engine(desc, 0)
    assert eng.force_form() is not None
    eng.energy(u, v)
    for atom in (0, n // 2, n - 1):  # its neighbours' indices above, on both sides of and below its own
        w = u.copy()
        w[atom, 2] += boxes * L
        with pytest.raises(nbg.EngineError) as ei:
            eng.energy(w, v)
        assert ei.value.status == -7  # NBG_ERR_RANGE
    # inside the cap a shifted image changes nothing but rounding
    w = u.copy()
    w[n // 2] += 1000 * L
    a, b = eng.energy(u, v)["potential"], eng.energy(w, v)["potential"]
    assert abs(a - b) <= 1e-9 * abs(a)
    eng.close()
