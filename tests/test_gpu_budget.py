"""Device memory under a budget: what the engine reports stays within it.

The budget covers the batch (wavefields, checkpoints or storage, the exact
adjoint's buffers) and what makes it faster -- event maps, the resident loops'
inbox, the second working buffer -- which is left out where it does not fit, with
the same bits.  Traces, residuals and observed data come on top.
"""
import numpy as np
import pytest

from cuda_fwi_gb300 import _capi
from cuda_fwi_gb300 import problem as P
from cuda_fwi_gb300.engine import Engine

pytestmark = pytest.mark.gpu


def _case(fwi=(1, 1, 1)):
    p = P.small(fdorder=4, nx=200, nz=200, nt=60, npml=20, nrec=6, perturb=0.04, seed=5, fwi=fwi)
    return p, np.random.default_rng(3).standard_normal((p.nrec, p.nt)) * 1e-2


def _run(p, obs, mode, snapshots, budget):
    with Engine(p) as e:
        e.set_gradient_mode(mode)
        e.set_strategy("binomial", snapshots=snapshots, budget_bytes=budget)
        rec, mis = e.forward([0], obs, keep=True)
        size = e.stats()["device_bytes"] - 3 * p.nrec * p.nt * 4
        launches = e.stats()["launches"]
        return [rec, mis, *e.backward()], size, launches


def _tightest(p, obs, mode, snapshots):
    """Smallest budget (to 256 bytes) that the engine takes."""
    lo, hi = 0, 1 << 30
    while hi - lo > 256:
        mid = (lo + hi) // 2
        try:
            _run(p, obs, mode, snapshots, mid)
            hi = mid
        except _capi.FwiError as ex:
            assert ex.code == "FWI_ERR_NOMEM"
            lo = mid
    return hi


@pytest.mark.parametrize("mode,fwi", [("reference", (1, 1, 1)), ("exact", (1, 1, 1)), ("exact", (1, 3, 2))])
def test_a_batch_stays_within_its_budget(mode, fwi):
    p, obs = _case(fwi)
    want, most, launches = _run(p, obs, mode, 4, 0)
    assert launches < p.nt  # the resident loop, whose inbox is reported
    b = _tightest(p, obs, mode, 4)
    assert b < most
    for budget in (b, (b + most) // 2, most):
        got, size, _ = _run(p, obs, mode, 4, budget)
        assert size <= budget
        for x, y in zip(got, want):
            assert np.array_equal(x, y)


def test_checkpoints_leave_room_for_the_loop():
    """As many checkpoints as the budget holds: a few less, and the loop still runs."""
    p, obs = _case()
    want, size, _ = _run(p, obs, "reference", 16, 0)
    got, held, launches = _run(p, obs, "reference", 0, size)
    assert held <= size and launches < p.nt
    for x, y in zip(got, want):
        assert np.array_equal(x, y)
