"""Gravity at the lines of its small-system forms: a body per thread up to 2048
padded bodies, the Morton order by counting up to 16,384 (blocks of 32 bodies,
2048 keys staged at a time, eight slices of them), a radix sort above; and
positions of which most share one Morton cell (ties keep the bodies' order)."""
import numpy as np
import pytest

import systems as S

nbg = S.nbg
pytestmark = pytest.mark.gpu

FORCE_TOL = 1e-5  # FP32 pair arithmetic with compensated positions, as everywhere


@pytest.mark.parametrize("far", [False, True], ids=["spread", "one-cell"])
@pytest.mark.parametrize("n, mass_spread", [(3, 0.0), (31, 0.5), (33, 0.0), (1793, 0.0), (2048, 0.5), (2049, 0.0), (4099, 0.5),
                                            (16384, 0.0), (16385, 0.0)])
def test_gravity_order_lines(gpu, oracle, n, mass_spread, far):
    sim = S.plummer(n, seed=n, mass_spread=mass_spread)
    desc, keep = nbg.system_descriptor(sim)
    u, v = S.state(sim)
    if far:
        u = u.copy()
        u[n // 2] = [3e6, -3e6, 3e6]  # one body so far away that its cube puts the others into a few cells
    eng = nbg.Engine(desc, 0)
    ag = eng.accel(v.copy(), u)
    ar, _ = oracle.accel(desc, v, u)
    assert S.rel_rmse(ag, ar) <= FORCE_TOL
    for _ in range(8):  # kept orders, then a sort with the kept extent buffer
        np.testing.assert_array_equal(eng.accel(v.copy(), u), ag)
    eng.close()
