"""Resident time loops (the default mapping on grids whose fields fit in the
SMs' shared memory) against the two-pass TMA tiles: the same arithmetic on
another schedule, so traces, misfits, wavefields, energies and checkpointed
gradients agree bit for bit.  With the wavefield stored, the two-pass mapping
takes its adjoint steps on the scalar cells, which round otherwise: there the
adjoint wavefield is compared with that of the two-pass checkpointed run (the
adjoint does not depend on where the forward fields come from), and the
gradient is bounded as between the other mappings (3e-5 relative L2).

The grids put the tile cuts where they can go wrong: one tile, tiles of the
least height, ragged widths and heights, strips over several tiles, a free
surface, several shots per launch and more shots than one launch holds.
"""
import numpy as np
import pytest

from conftest import rel_l2
from cuda_fwi_gb300 import problem as P
from cuda_fwi_gb300.engine import Engine

pytestmark = pytest.mark.gpu

CASES = [
    # order, nx, nz, npml, fsurf, shots, nt
    (2, 30, 21, 0, 0, 1, 60),
    (2, 61, 47, 5, 1, 3, 90),
    (4, 200, 200, 20, 0, 1, 150),
    (4, 97, 333, 11, 1, 2, 100),
    (6, 131, 60, 9, 1, 5, 100),
    (8, 150, 50, 8, 0, 2, 120),
    (8, 513, 290, 30, 0, 1, 90),
    (4, 295, 112, 12, 0, 35, 40),
    (10, 120, 90, 12, 0, 2, 90),
    (12, 403, 101, 24, 1, 3, 80),
]


def _case(order, nx, nz, npml, fsurf, shots, nt, fwi=(1, 1, 1)):
    kw = dict(fdorder=order, nx=nx, nz=nz, nt=nt, npml=npml, fsurf=fsurf, nshots=shots, nrec=9, fwi=fwi)
    p = P.small(seed=3, perturb=0.05, **kw)
    obs = np.random.default_rng(7).standard_normal((p.nrec, nt)) * 1e-2
    return p, obs


def _run(p, obs, bx, strategy, graphs=True):
    shots = list(range(p.nshots))
    with Engine(p) as e:
        e.set_exec(graphs, bx, 0)
        if strategy == "binomial":
            e.set_strategy("binomial", snapshots=5)
        rec, mis = e.forward(shots, obs, keep=True)
        launches = e.stats()["launches"]
        w = [e.wavefield(0, b) for b in (0, p.nshots - 1)]
        g = e.backward()
        wa = [e.wavefield(1, b) for b in (0, p.nshots - 1)]
        en = [e.energy(b) for b in (0, p.nshots - 1)]
    return dict(rec=rec, mis=mis, w=w, g=g, wa=wa, en=en, launches=launches)


@pytest.mark.parametrize("case", CASES, ids=lambda c: "o%d_%dx%d_p%d_fs%d_s%d" % c[:6])
@pytest.mark.parametrize("strategy", ["binomial", "full"])
def test_resident_loops_equal_the_two_pass_tiles(case, strategy):
    p, obs = _case(*case, fwi=(1, 1, 1) if strategy == "binomial" else (2, 1, 3))
    a, b = _run(p, obs, 0, strategy), _run(p, obs, 256, strategy)
    assert a["launches"] < b["launches"]  # the loop ran in one launch (per group of shots)
    assert np.array_equal(a["rec"], b["rec"]) and np.array_equal(a["mis"], b["mis"])
    adj = b if strategy == "binomial" else _run(p, obs, 256, "binomial")
    for k, ref in (("w", b), ("wa", adj)):
        for x, y in zip(a[k], ref[k]):
            for f in x:
                assert np.array_equal(x[f], y[f]), (k, f)
    for x, y in zip(a["en"], adj["en"]):
        assert np.array_equal(x[0], y[0]) and np.array_equal(x[1], y[1])
    for x, y in zip(a["g"], b["g"]):
        if strategy == "binomial":
            assert np.array_equal(x, y)
        else:
            assert rel_l2(x, y) <= 3e-5


def test_resident_loops_repeat_and_follow_a_changed_batch():
    """The same engine on other shots, then the first ones again: nothing carries over."""
    p, obs = _case(8, 150, 50, 8, 0, 4, 80)
    with Engine(p) as e:
        e.set_strategy("binomial", snapshots=4)
        first = e.gradient([0, 1], obs)
        e.gradient([2, 3, 1], obs)
        e.misfit([3], obs)
        again = e.gradient([0, 1], obs)
    for x, y in zip(first[0], again[0]):
        assert np.array_equal(x, y)
    assert np.array_equal(first[1], again[1])


@pytest.mark.parametrize("grid,backward_resident", [((4, 200, 200, 20), True), ((8, 600, 380, 20), False)],
                         ids=["both_sweeps", "forward_only"])
def test_a_changed_sampling_interval_changes_the_programs(grid, backward_resident):
    """One engine through several FWI intervals (the number of checkpoints stays, so
    does the number of saves of the forward sweep) gives what a fresh one gives."""
    order, nx, nz, npml = grid
    p, obs = _case(order, nx, nz, npml, 0, 1, 120)

    def run(e, interval):
        e.set_fwi(interval, 1, 1)
        rec, mis = e.forward([0], obs, keep=True)
        assert e.stats()["launches"] < p.nt
        g = e.backward()
        assert (e.stats()["launches"] < p.nt) == backward_resident
        return [rec, mis, *g]

    def engine():
        e = Engine(p)
        e.set_strategy("binomial", snapshots=5)
        return e

    with engine() as e:
        for interval in (2, 1, 3, 1, 2):
            with engine() as fresh:
                want = run(fresh, interval)
            for a, b in zip(run(e, interval), want):
                assert np.array_equal(a, b), interval


@pytest.mark.parametrize("grid,shots", [((8, 400, 300, 20), 8), ((6, 300, 300, 20), 16), ((12, 150, 150, 20), 24)])
def test_stored_gradient_does_not_depend_on_the_batch(grid, shots):
    """A shot's gradient over a stored wavefield is the same bits alone and among many."""
    order, nx, nz, npml = grid
    p, obs = _case(order, nx, nz, npml, 0, shots, 90)
    with Engine(p) as e:
        e.set_strategy("full")
        rec, mis = e.forward(list(range(shots)), obs, keep=True)
        g = e.backward()
        for s in (0, shots - 1):
            _, m1 = e.forward([s], obs, keep=True)
            assert m1[0] == mis[s]
            for a, b in zip(e.backward(), g):
                assert np.count_nonzero(a[0]) and np.array_equal(a[0], b[s])
