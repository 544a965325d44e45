"""Checkpointed backward with the recomputed forward steps on a stream of their own.

Where the memory budget has no room for the second working buffer the same plan
runs on one stream: both give the same seismograms and gradients bit for bit, for
few and many checkpoints (plans that restore the zero state, that take a state
from a slot straight to its adjoint step, that save into a slot just read), with
graphs and direct launches, for one and several shots, sampled steps and the
widest halo, and again on a second call.
"""
import numpy as np
import pytest

from cuda_fwi_gb300 import _capi
from cuda_fwi_gb300 import problem as P
from cuda_fwi_gb300.engine import Engine

pytestmark = pytest.mark.gpu


def _tightest(e, snapshots, run):
    """Smallest budget (to 256 bytes) that the engine takes with these checkpoints."""
    lo, hi = 0, 1 << 30
    while hi - lo > 256:
        mid = (lo + hi) // 2
        e.set_strategy("binomial", snapshots=snapshots, budget_bytes=mid)
        try:
            run()
            hi = mid
        except _capi.FwiError as ex:
            assert ex.code == "FWI_ERR_NOMEM"
            lo = mid
    return hi


@pytest.mark.parametrize("mode", ["reference", "exact"])
@pytest.mark.parametrize("order,shots,slots,sample,graphs",
                         [(4, 1, 1, 1, True), (8, 1, 3, 1, False), (8, 3, 7, 1, True), (12, 2, 4, 1, True),
                          (2, 2, 5, 2, False), (6, 1, 60, 1, True)])
def test_two_streams_agree_with_one(order, shots, slots, sample, graphs, mode):
    sample = 1 if mode == "exact" else sample
    p = P.small(fdorder=order, nx=150, nz=60, nt=64, npml=8, nshots=shots, nrec=6, perturb=0.04, seed=21,
                fwi=(sample, 1, 1))
    obs = np.random.default_rng(4).standard_normal((p.nrec, p.nt)) * 1e-6
    ids = list(range(shots))
    out, size = [], []
    for tight in (False, True):
        with Engine(p) as e:
            e.set_exec(graphs, 256, 0)  # launches per pass, not the resident loops
            e.set_gradient_mode(mode)
            e.set_strategy("binomial", snapshots=slots)
            if tight:
                b = _tightest(e, slots, lambda: e.forward(ids, obs, keep=True))
        with Engine(p) as e:
            e.set_exec(graphs, 256, 0)
            e.set_gradient_mode(mode)
            e.set_strategy("binomial", snapshots=slots, budget_bytes=b if tight else 0)
            for _ in range(2):
                rec, mis = e.forward(ids, obs, keep=True)
                g = e.backward()
                out.append((rec, mis, *g))
            size.append(e.stats()["device_bytes"])
    assert size[0] > size[1]  # the second working buffer is there, and is not
    for run in out[1:]:
        for a, b in zip(out[0], run):
            assert np.array_equal(a, b)
