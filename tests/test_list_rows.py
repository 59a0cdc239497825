"""Capacities of the Verlet-list rows: whole 16-byte units from the first one
through every growth (the force kernels' tensor map and the replica loop's
16-byte loads need them), and a replica batch whose rows grow twice, against
the FP64 oracle."""
import os
import subprocess

import numpy as np
import pytest

import systems as S

nbg = S.nbg
CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "nbodysimulator.jl_gb300", "csrc")

PROGRAM = r"""
#include <cstdio>
#include "list_rows.h"
int main()
{
    for (int wanted = 1; wanted <= 1200; ++wanted) {
        int cap = list_row_capacity(wanted);
        std::printf("%d", wanted);
        for (int k = 0; k < 8; ++k, cap = list_grown_capacity(cap)) std::printf(" %d", cap);
        std::printf("\n");
    }
}
"""


def test_row_capacities_stay_whole(tmp_path):
    src, exe = tmp_path / "rows.cpp", tmp_path / "rows"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-I", CSRC, str(src), "-o", str(exe)], check=True)
    rows = [list(map(int, line.split())) for line in subprocess.run([str(exe)], check=True, capture_output=True,
                                                                    text=True).stdout.splitlines()]
    assert len(rows) == 1200
    for wanted, *caps in rows:
        assert caps[0] >= wanted and caps[0] - wanted < max(8, 33 - wanted)
        for c in caps:
            assert c % 8 == 0
            # the replica loop's blocks of 8 entries per lane, 4 or 8 lanes
            for lanes in (4, 8):
                assert -(-c // (8 * lanes)) * 8 * lanes <= 2 * c
        for a, b in zip(caps, caps[1:]):
            assert b >= a + a // 2 + 32 and b - (a + a // 2 + 32) < 8


def _droplets(lanes, monkeypatch):
    """Replicas that are a dense droplet each in a wide box: 90 and more
    neighbours where the mean density gives fewer than four."""
    if lanes:
        monkeypatch.setenv("NBG_LIST_LPA", str(lanes))
    descs, keep, us, vs = [], [], [], []
    for r, side in enumerate((5, 6, 7)):
        n, L = side ** 3, 24.0
        g = np.arange(side) * (0.95 + 0.02 * r) + 5.0
        rng = np.random.default_rng(r)
        u = np.stack(np.meshgrid(g, g, g, indexing="ij"), -1).reshape(-1, 3) + rng.uniform(-0.02, 0.02, (n, 3))
        d, k = nbg.lennard_jones_descriptor(np.ones(n), L, skin=0.5, seed=r, thermostat=nbg.LangevinThermostat(0.7, 1.0))
        d.flags |= nbg._abi.NBG_FLAG_LANGEVIN_BAOAB
        descs.append(d)
        keep.append(k)
        us.append(u)
        vs.append(rng.standard_normal((n, 3)) * 0.8)
    return descs, keep, np.concatenate(us), np.concatenate(vs)


# lanes per atom of the batch's step graphs: as chosen (one here: nothing else
# looks at the rows' alignment), 4, and 32
@pytest.mark.gpu
@pytest.mark.parametrize("lanes", [0, 4, 32])
def test_batch_whose_rows_grow_twice(gpu, oracle, monkeypatch, lanes):
    descs, keep, u, v = _droplets(lanes, monkeypatch)
    eng = nbg.Engine(descs, 0)
    assert eng.ensemble_form() is not None
    if not lanes:
        assert eng.force_form()[0] == 1
    ug, vg, _, _, _ = eng.run(u, v, 0.002, 25, 0, save_trajectory=False, step=0)
    ag = eng.get_accel()
    eng.close()
    off = 0
    for d in descs:
        n = int(d.n)
        s = slice(off, off + n)
        # (more neighbours than the first capacity, 40, and the next one, 96, hold)
        dx = u[s][:, None] - u[s][None]
        assert (np.sum(dx * dx, axis=2) < 3.0 ** 2).sum(axis=1).max() - 1 > 96
        ao, _ = oracle.accel(d, vg[s].copy(), ug[s])
        assert S.rel_rmse(ag[s], ao) <= 1e-5  # FP32 pair arithmetic, as everywhere
        off += n
