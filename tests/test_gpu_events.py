"""Injection and recording inside the velocity passes: cells with several events
(two sources and three receivers on one cell, receivers on neighbouring cells),
and events spread over more rows than an event map covers.

The order of a cell's events is part of the result (sources in index order, then
the receivers), so the launches per pass and the resident time loops agree bit
for bit, and both match the FP64 oracle (seismograms 1e-5, gradients 1e-4
relative L2, as everywhere).
"""
import numpy as np
import pytest

from conftest import rel_l2
from cuda_fwi_gb300 import problem as P
from cuda_fwi_gb300.engine import Engine
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _crowded(order, fsurf):
    p = P.small(fdorder=order, nx=70, nz=44, nt=120, npml=8, fsurf=fsurf, nrec=4, perturb=0.04, seed=5)
    p.set_sources([30, 30, 31, 44], [6, 6, 6, 20], [0, 0, 0, 0], [15.0, 11.0, 13.0, 9.0])
    p.set_receivers([30, 30, 30, 31, 32, 33, 44, 60, 61], [6, 6, 6, 6, 6, 7, 20, 20, 20], np.zeros(9, np.int32))
    return p


@pytest.mark.parametrize("order,fsurf", [(4, 0), (8, 1)])
def test_several_events_in_a_cell(order, fsurf):
    p = _crowded(order, fsurf)
    obs = np.random.default_rng(1).standard_normal((p.nrec, p.nt)) * 1e-2
    J, g_o, fw_o, _ = O.gradient(p, obs, 0)
    out = []
    for bx in (0, 256):
        with Engine(p) as e:
            e.set_exec(True, bx, 0)
            e.set_strategy("binomial", snapshots=5)
            rec, mis = e.forward([0], obs, keep=True)
            g = e.backward()
        assert rel_l2(rec[: p.nrec], fw_o["rec"]) <= 1e-5
        assert mis[0] == pytest.approx(J, rel=1e-4)
        for i in range(3):
            assert rel_l2(g[i][0], g_o[i]) <= 1e-4
        out.append((rec, *[x[0] for x in g]))
    for a, b in zip(*out):
        assert np.array_equal(a, b)


def test_events_over_many_rows():
    """A receiver in every row: the maps of three shots together are too large, one shot's is not."""
    p = P.small(fdorder=4, nx=480, nz=380, nt=40, npml=10, nshots=3, nrec=6, perturb=0.04, seed=9)
    z = np.arange(2, 378)
    n = len(z)
    p.set_receivers(np.tile(np.full(n, 200), 3), np.tile(z, 3), np.repeat(np.arange(3, dtype=np.int32), n))
    obs = np.random.default_rng(2).standard_normal((p.nrec, p.nt)) * 1e-2
    with Engine(p) as e:
        e.set_exec(True, 256, 0)
        e.set_strategy("binomial", snapshots=4)
        rec, mis = e.forward([0, 1, 2], obs, keep=True)
        g = e.backward()
        for s in range(3):
            r1, m1 = e.forward([s], obs, keep=True)
            g1 = e.backward()
            rows = O.shot_rows(p, s)
            assert np.array_equal(r1[rows], rec[rows]) and m1[0] == mis[s]
            for q in range(3):
                assert np.array_equal(g1[q][0], g[q][s])


@pytest.mark.parametrize("order,nt", [(4, 12), (8, 13)])
def test_energy_of_two_steps_at_once(order, nt):
    """A large launch adds the energies of two steps at once, a launch of one of its
    shots each step's: the same sums, in cells with sources and residuals too (the
    last shot's sources share receivers' cells), for an odd and an even nt."""
    n = 12
    p = P.small(fdorder=order, nx=960, nz=500, nt=nt, npml=16, nshots=n, nrec=5, perturb=0.04, seed=7)
    p.set_sources([300] * (n - 1) + [30, 30, 31, 44], [20] * (n - 1) + [6, 6, 6, 20],
                  list(range(n - 1)) + [n - 1] * 4, 15.0)
    rx = [30, 30, 31, 32, 44, 300, 301]
    rz = [6, 6, 6, 6, 20, 20, 20]
    p.set_receivers(np.tile(rx, n), np.tile(rz, n), np.repeat(np.arange(n, dtype=np.int32), len(rx)))
    obs = np.random.default_rng(6).standard_normal((p.nrec, nt)) * 1e-2
    with Engine(p) as e:
        e.set_strategy("binomial", snapshots=4)
        e.forward(list(range(n)), obs, keep=True)
        e.backward()
        all_shots = [e.energy(k) for k in (0, n - 1)]
        for k, want in zip((0, n - 1), all_shots):
            e.forward([k], obs, keep=True)
            e.backward()
            got = e.energy(0)
            for a, b in zip(got, want):
                assert np.count_nonzero(a) and np.array_equal(a, b)
