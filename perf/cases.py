"""Workloads of the elastic P-SV engine, for timing it through its public entry points.

Each case is one call (or the forward/backward pair) that a modelling or inversion
program makes again and again: a new earth model goes in (device tensors, or host
arrays where the entry point takes those), traces, misfits and gradients come out.

Grids, orders, CPML widths, receiver counts and strategies are those of the
package's own workloads (200x200 order 4, 800x400 order 8, 1000x500 order 8 with
64 shots, uneven models of orders 4 and 8, 2000x600 order 8 with 96 shots) and of
its tests (orders 2..12, free surface, sampled windows).  Records are shorter than
a production record (nt 1000-5000): the cost per time step does not depend on nt,
and the checkpoint counts are lowered with nt so that the recomputed steps per
recorded step stay what they are for 32 checkpoints over 3000 steps (about 1.8).

Observed records are hyperbolic arrivals (a direct wave and reflections), so the
residual is of the size of the data, as it is when an inversion starts.

The engine computes in FP32 and hands its results over as FP64 host arrays in
the reference's layouts; the program keeps them as what they hold, FP32.
"""
import math
import random

import numpy as np
import torch

from cuda_fwi_gb300 import _capi
from cuda_fwi_gb300.autograd import FWIMisfit
from cuda_fwi_gb300.engine import Engine
from cuda_fwi_gb300.multi import MultiEngine
from cuda_fwi_gb300.problem import Problem


def _case(name, kind, nx, nz, order, npml, nt, shots, nrec, fsurf=0, slots=0, sample=1):
    return {"name": name, "kind": kind, "nx": nx, "nz": nz, "order": order, "npml": npml, "nt": nt,
            "shots": shots, "nrec": nrec, "fsurf": fsurf, "slots": slots, "sample": sample}


def listed():
    return [
        # modelling one shot on a small grid: every launch counts
        _case("model_200x200_1shot", "forward", 200, 200, 4, 20, 300, 1, 50),
        # the plain gradient: one shot, the whole forward wavefield stored, forward and backward calls
        _case("stored_gradient_200x200", "stored", 200, 200, 4, 20, 1000, 1, 50),
        # stored gradient on a sampled window (every second step, row and column), order 2, ragged grid
        _case("stored_sampled_399x301_o2", "stored", 399, 301, 2, 15, 300, 2, 100, sample=2),
        # checkpointed gradient of a few shots under a free surface, ragged grid, order 6
        _case("gradient_fsurf_501x243_o6", "gradient", 501, 243, 6, 20, 240, 3, 120, fsurf=1, slots=10),
        # the differentiable misfit (exact discrete adjoint) on the 800x400 grid, host tensors in and out
        _case("autograd_exact_800x400", "exact", 800, 400, 8, 30, 120, 1, 200, slots=8),
        # one shot of the large grid: the reference's update after every shot
        _case("gradient_2000x600_1shot", "gradient", 2000, 600, 8, 40, 100, 1, 400, slots=6),
        # the batched multi-shot gradient, the package's headline workload
        _case("gradient_1000x500_64shots", "gradient", 1000, 500, 8, 30, 160, 64, 250, slots=8),
        # a trial misfit of the step-length search: forward only, many shots of the large grid
        _case("misfit_2000x600_96shots", "misfit", 2000, 600, 8, 40, 60, 96, 400),
        # high order, wide halo, a handful of shots with their traces
        _case("model_403x307_o12_6shots", "forward", 403, 307, 12, 24, 200, 6, 150, fsurf=1),
        # independent models of uneven size and record length in one launch
        _case("uneven_8models", "uneven", 1200, 600, 8, 30, 240, 8, 0, slots=10),
        # the reference's own call pair: host FP64 arrays, storage handed back and in again
        _case("reference_call_100x80_o2", "reference", 100, 80, 2, 12, 120, 1, 24),
    ]


# cost of a case in cell-steps (recompute, adjoint and correlation included), for keeping draws small
_WEIGHT = {"forward": 1.0, "misfit": 1.0, "stored": 4.0, "gradient": 5.0, "exact": 9.0, "uneven": 5.0, "reference": 12.0}


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["forward", "forward", "stored", "gradient", "gradient", "gradient", "misfit", "exact", "uneven",
                       "reference"])
    order = rng.choice([2, 4, 4, 6, 8, 8, 8, 10, 12])
    npml = rng.randint(10, 40)
    nx, nz = _log(rng, 100, 2000), _log(rng, 80, 600)
    nt = _log(rng, 60, 500)
    shots = _log(rng, 1, 64)
    sample = 1
    if kind == "stored":
        nx, nz, shots = min(nx, 500), min(nz, 400), min(shots, 4)
        sample = rng.choice([1, 1, 2, 3])
    if kind == "exact":
        nx, nz, nt, shots = min(nx, 800), min(nz, 400), min(nt, 160), min(shots, 2)
    if kind == "reference":
        nx, nz, nt, shots, order = min(nx, 160), min(nz, 120), min(nt, 150), 1, rng.choice([2, 4])
    if kind == "uneven":
        nx, nz, order, npml, shots = max(nx, 240), max(nz, 220), 8, 30, rng.randint(3, 10)
    limit = 8e9  # cell-steps: the largest listed case has 3e10
    while _WEIGHT[kind] * (nx + 2 * npml) * (nz + 2 * npml) * nt * shots > limit:
        if shots > 1:
            shots = max(1, shots // 2)
        else:
            nt = max(40, nt // 2)
    slots = rng.randint(max(3, nt // 40), max(4, nt // 12)) if kind in ("gradient", "exact", "uneven") else 0
    fsurf = int(kind != "uneven" and rng.random() < 0.35)
    c = _case("", kind, nx, nz, order, npml, nt, shots, max(4, nx // rng.randint(3, 8)), fsurf, slots, sample)
    del c["name"]
    return c


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
DX, DT = 10.0, 1e-3  # m, s


def _models(c):
    """The grids of a case: (nx, nz, order, nt, nrec) per model (one, but for the uneven batch)."""
    if c["kind"] != "uneven":
        return [(c["nx"], c["nz"], c["order"], c["nt"], c["nrec"])]
    r = random.Random(c["nx"] * 131 + c["nz"])  # the sizes belong to the case, not to the seed
    out = []
    for k in range(c["shots"]):
        nx, nz = r.randint(200, c["nx"]), r.randint(200, c["nz"])
        out.append((nx, nz, (4, 8)[k % 2] if k < 2 else r.choice([4, 8]), r.randint(max(40, c["nt"] // 3), c["nt"]),
                    max(2, nx // 4)))
    return out


def _padding(c, order):
    """fpad, ppad, rows above the model in the padded grid."""
    fpad = order // 2
    ppad = c["npml"] + fpad
    return fpad, ppad, fpad if c["fsurf"] else ppad


def _earth(c, nx, nz, order, rng):
    """lam, mu, rho [nzt][nxt] FP64: six layers 1800..4500 m/s with a smooth +-3 % perturbation, Gardner density."""
    fpad, ppad, ztop = _padding(c, order)
    z, x = np.arange(nz)[:, None], np.arange(nx)[None, :]
    edges = np.linspace(0, nz, 7)[1:-1] + rng.uniform(-0.04, 0.04, 5) * nz
    vp = np.linspace(1800.0, 4500.0, 6)[np.searchsorted(edges, np.arange(nz), side="right")][:, None]
    p = np.zeros((nz, nx))
    for _ in range(6):
        kz, kx = rng.uniform(0.01, 0.15, 2)
        p += np.cos(kz * z + rng.uniform(0, 6.28)) * np.cos(kx * x + rng.uniform(0, 6.28))
    vp = vp * (1.0 + 0.03 * p / np.abs(p).max())
    vs, rho = vp / 1.73, 310.0 * vp ** 0.25
    pads = ((ztop, ppad), (ppad, ppad))
    mu, rho = np.pad(vs * vs * rho, pads, mode="edge"), np.pad(rho, pads, mode="edge")
    lam = np.pad(vp * vp * (310.0 * vp ** 0.25), pads, mode="edge") - 2.0 * mu
    return [np.ascontiguousarray(a) for a in (lam, mu, rho)]


def _ricker(nt, f0, shift):
    t = np.arange(nt) * DT
    tau = np.pi * (t - 1.5 / f0 - shift) / (1.5 / f0)
    return (1.0 - 2.0 * tau * tau) * np.exp(-2.0 * tau * tau)


def _observed(src_x, rec_x, nt, rng):
    """[len(src_x) * len(rec_x)][nt]: a direct arrival and three reflections with hyperbolic moveout."""
    off = np.abs(src_x[:, None] - rec_x[None, :]).reshape(-1, 1) * DX
    t = np.arange(nt)[None, :] * DT
    obs = np.zeros((off.shape[0], nt))
    for k in range(4):
        v, t0 = rng.uniform(1700.0, 4200.0), nt * DT * (0.05 if k == 0 else rng.uniform(0.2, 0.8))
        arg = (math.pi * 12.0) ** 2 * (t - np.sqrt(t0 * t0 + (off / v) ** 2)) ** 2
        obs += 0.02 * rng.uniform(0.5, 1.5) * (1.0 - 2.0 * arg) * np.exp(-arg) / (1.0 + off / 200.0)
    return obs


def _inputs(c, seed):
    """Per model of the case: earth, acquisition (model coordinates), signals and observed records, from the seed alone."""
    rng = np.random.default_rng([seed, c["nx"], c["nz"], c["nt"]])
    out = []
    for nx, nz, order, nt, nrec in _models(c):
        earth = _earth(c, nx, nz, order, rng)
        n = 1 if c["kind"] == "uneven" else c["shots"]
        f0 = rng.uniform(10.0, 15.0)
        sx = np.linspace(4, nx - 5, n).round().astype(np.int32) if n > 1 else np.array([nx // 2 + rng.integers(-3, 4)], np.int32)
        rx = np.linspace(0, nx - 1, nrec).round().astype(np.int32)
        # the wavelet starts shortly before its peak, so that a short record holds waves
        sig = _ricker(nt, f0, -0.9 / f0)
        out.append({"earth": earth, "order": order, "nx": nx, "nz": nz, "nt": nt, "sx": sx, "sz": 5, "rx": rx, "rz": 5,
                    "shots": n, "sig": sig, "f0": f0, "obs": _observed(sx, rx, nt, rng)})
    return out


def _problem(c, m):
    p = Problem(nx=m["nx"], nz=m["nz"], nt=m["nt"], dx=DX, dz=DX, dt=DT, fdorder=m["order"], npml=c["npml"],
                fsurf=c["fsurf"], fpml=10.0, damp_v_pml=4500.0, fwi_dt=c["sample"], fwi_dx=c["sample"],
                fwi_dz=c["sample"]).finalize()
    n, nr = m["shots"], len(m["rx"])
    p.set_sources(m["sx"], np.full(n, m["sz"]), np.arange(n), m["f0"], ts=-0.9 / m["f0"])
    p.set_receivers(np.tile(m["rx"], n), np.full(n * nr, m["rz"]), np.repeat(np.arange(n, dtype=np.int32), nr))
    p.lam, p.mu, p.rho = m["earth"]
    return p


def prepare(case, seed):
    ins = _inputs(case, seed)
    kind = case["kind"]
    s = {"kind": kind, "shots": list(range(ins[0]["shots"])), "obs": ins[0]["obs"]}
    ps = [_problem(case, m) for m in ins]
    if kind == "uneven":
        s["engine"] = MultiEngine(ps, snapshots=case["slots"])
        s["obs"] = [m["obs"] for m in ins]
        return s
    p = ps[0]
    if kind == "reference":
        return dict(s, **_reference_arrays(p))
    s["engine"] = e = Engine(p, set_model=False)
    if kind in ("gradient", "exact"):
        e.set_strategy("binomial", snapshots=case["slots"])
    elif kind == "stored":
        e.set_strategy("full")
    if kind == "exact":
        s["model"] = [torch.from_numpy(a).requires_grad_() for a in ins[0]["earth"]]
    else:
        s["model"] = [torch.from_numpy(a).cuda() for a in ins[0]["earth"]]
    return s


def _reference_arrays(p):
    """What a caller of the reference's propagator pair holds: its host arrays."""
    tp = 2 * (p.npml + 1)
    xs, zs = lambda: np.zeros((p.nzt, tp)), lambda: np.zeros((tp, p.nxt))  # noqa: E731
    return {"p": p, "avg": _capi.average_parameters(p.mu, p.rho),
            "wave": [[np.zeros((p.nzt, p.nxt)) for _ in range(6)] for _ in range(2)],
            "mem": [xs(), zs(), xs(), zs(), xs(), xs(), zs(), zs()],
            "cp": [np.ascontiguousarray(p.cpml[k]) for k in ("a", "b", "K", "a_half", "b_half", "K_half")],
            "rec": np.zeros((p.nrec, p.nt)), "store": [np.zeros((p.nft, p.nfz, p.nfx)) for _ in range(5)],
            "grad": [np.zeros((p.nfz, p.nfx)) for _ in range(3)]}


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def _f32(a):
    return np.asarray(a).astype(np.float32)


def run(state):
    kind, e = state["kind"], state.get("engine")
    if kind == "uneven":
        g, mis = e.gradient(state["obs"])
        return {"misfit": _f32(mis), "grad": [[_f32(a) for a in t] for t in g]}
    if kind == "reference":
        return _run_reference(state)
    if kind == "exact":
        lam, mu, rho = state["model"]
        for t in state["model"]:
            t.grad = None
        j = FWIMisfit.apply(lam, mu, rho, e, state["shots"], state["obs"], "exact")
        j.backward()
        return {"misfit": j.detach().float(), "grad": [t.grad.float() for t in state["model"]]}
    e.set_model_device(*state["model"])
    if kind == "forward":
        rec, _ = e.forward(state["shots"])
        return {"rec": _f32(rec)}
    if kind == "misfit":
        return {"misfit": _f32(e.misfit(state["shots"], state["obs"]))}
    if kind == "stored":
        rec, mis = e.forward(state["shots"], state["obs"], keep=True)
        g = e.backward()
        return {"rec": _f32(rec), "misfit": _f32(mis), "grad": [_f32(a) for a in g]}
    g, mis = e.gradient(state["shots"], state["obs"])
    return {"misfit": _f32(mis), "grad": [_f32(a) for a in g]}


def _run_reference(s):
    p, pd, pi, lib = s["p"], _capi.pd, _capi.pi, _capi.lib()
    mz, rz, rx = s["avg"]
    grid = (0, p.nt, p.nzt, p.nxt, p.fpad, p.ppad, p.dt, p.dx, p.dz, p.nt, p.fsurf, pd(p.hc), p.fdorder)
    mat = [pd(a) for a in (p.lam, p.mu, mz, rz, rx)]
    cpml = [p.npml, *[pd(a) for a in s["cp"]], *[pd(a) for a in s["mem"]]]
    win = (1, p.fwi_dt, p.fwi_dx, p.fwi_dz, p.x1, p.x2, p.z1, p.z2)
    recv = (p.nrec, pi(p.rec_x), pi(p.rec_z), pi(p.rec_comp))
    _capi.check(lib.fwi_psv_forward_kernel(
        *grid, *[pd(a) for a in s["wave"][0]], *mat, *cpml, p.nsrc, pi(p.src_x), pi(p.src_z), pi(p.src_comp),
        pd(p.src_signal), pi(p.src_shot), *recv, pd(s["rec"]), pi(p.rec_shot), *win, *[pd(a) for a in s["store"]]),
        "forward_kernel")
    residual = s["rec"] - s["obs"]
    _capi.check(lib.fwi_psv_adjoint_kernel(
        *grid, *[pd(a) for a in s["wave"][1]], *mat, *cpml, *recv, pd(residual), pi(p.rec_shot), *win,
        *[pd(a) for a in s["store"]], *[pd(a) for a in s["grad"]]), "adjoint_kernel")
    return {"rec": _f32(s["rec"]), "grad": [_f32(a) for a in s["grad"]],
            "forward": [_f32(a) for a in s["wave"][0][:5]], "adjoint": [_f32(a) for a in s["wave"][1][:5]]}


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def work(case):
    """Per cell and time step in FP32: the five fields read and written once by the forward step (40 bytes) and by the
    adjoint step (40), whose correlation reads the five forward fields (20) and updates ux, uz and three gradients
    (40); a stored wavefield is also written once (20).  The forward steps that a checkpointed pass recomputes are not
    counted.  Operations: eight derivatives of order / 2 taps (three each) and the updates."""
    b = f = 0.0
    for nx, nz, order, nt, nrec in _models(case):
        fpad, ppad, ztop = _padding(case, order)
        cells = (nx + 2 * ppad) * (nz + ppad + ztop)
        steps = float(cells) * nt * (1 if case["kind"] == "uneven" else case["shots"])
        flops = 8 * 1.5 * order + 14
        b += 40 * steps + 5 * 4 * cells
        f += flops * steps
        if case["kind"] not in ("forward", "misfit"):
            k = case["sample"]
            b += (56 + 64.0 / k ** 3) * steps
            f += (flops + 4 + 30.0 / k ** 3) * steps
    return {"bytes": b, "flops": f}


# ---------------------------------------------------------------------------
# the same in 64 bits, from the scheme's formulas
# ---------------------------------------------------------------------------
# Holberg's optimised staggered-grid coefficients (maximum group-velocity error 0.1 %), orders 2..12
_HOLBERG = {2: [1.0010], 4: [1.1382, -0.046414], 6: [1.1965, -0.078804, 0.0081781],
            8: [1.2257, -0.099537, 0.018063, -0.0026274],
            10: [1.2415, -0.11231, 0.026191, -0.0064682, 0.001191],
            12: [1.2508, -0.12034, 0.032131, -0.010142, 0.0029857, -0.00066667]}


def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _cpml_lines(npml, fpad, n, low):
    """a, b, 1/K (integer and half points) along an axis of n interior cells, layers at the low (if `low`) and high end."""
    thick, alpha_max = npml * DX, math.pi * 10.0
    d0 = -3.0 * 4500.0 * math.log(1e-3) / (2.0 * thick)
    c = {k: torch.zeros(n, dtype=torch.float64) for k in ("a", "b", "ah", "bh")}

    def put(i, dist, a, b):
        if dist < 0:
            return
        xn = dist / thick
        d, al = d0 * xn * xn, max(0.0, alpha_max * (1.0 - xn))
        c[b][i] = math.exp(-(d + al) * DT)
        if abs(d) > 1e-6:
            c[a][i] = d * (c[b][i] - 1.0) / (d + al)

    if low:
        for k in range(npml):
            put(k, thick - k * DX, "a", "b")
            put(k, thick - (k + 0.5) * DX, "ah", "bh")
    deep = npml if low else npml + 1  # under a free surface the bottom layer is one cell deeper
    for k in range(deep):
        put(n - deep + k, k * DX, "a", "b")
        put(n - deep + k, (k + 0.5) * DX, "ah", "bh")
    return c


class _Scheme:
    """One time step of the staggered scheme for a stack of shots [shot][nzt][nxt], on new tensors."""

    def __init__(self, c, m, earth):
        self.dev = earth[0].device
        self.fpad, self.ppad, _ = _padding(c, m["order"])
        self.fsurf, self.npml = c["fsurf"], c["npml"]
        self.nzt, self.nxt = earth[0].shape
        self.h = [v / DX for v in _HOLBERG[m["order"]]]
        lam, mu, rho = earth
        F = self.fpad
        inner = (slice(F, self.nzt - F), slice(F, self.nxt - F))
        self.inner = inner
        right, down = torch.roll(mu, -1, 1), torch.roll(mu, -1, 0)
        muzx = 4.0 / (1.0 / mu + 1.0 / right + 1.0 / down + 1.0 / torch.roll(right, -1, 0))
        self.lam, self.mu, self.muzx = lam[inner], mu[inner], muzx[inner]
        self.bx = (2.0 / (rho + torch.roll(rho, -1, 1)))[inner]
        self.bz = (2.0 / (rho + torch.roll(rho, -1, 0)))[inner]
        lines = [_cpml_lines(self.npml, F, self.nxt - 2 * F, True), _cpml_lines(self.npml, F, self.nzt - 2 * F, not c["fsurf"])]
        self.px = {k: v.to(self.dev)[None, None, :] for k, v in lines[0].items()}
        self.pz = {k: v.to(self.dev)[None, :, None] for k, v in lines[1].items()}

    def start(self, shots):
        z = torch.zeros(shots, self.nzt, self.nxt, dtype=torch.float64, device=self.dev)
        q = torch.zeros(shots, self.nzt - 2 * self.fpad, self.nxt - 2 * self.fpad, dtype=torch.float64, device=self.dev)
        return [z] * 5 + [q] * 8  # vx vz sxx szx szz, then the CPML memories

    def diff(self, f, axis, up):
        """sum_k h_k (f[c+k-1] - f[c-k]), or one point further with `up`, on the interior."""
        F, n = self.fpad, f.shape[axis]
        other = 3 - axis
        f = f.narrow(other, F, f.shape[other] - 2 * F)
        d = 0
        for k in range(1, F + 1):
            a, b = (k, 1 - k) if up else (k - 1, -k)
            d = d + self.h[k - 1] * (f.narrow(axis, F + a, n - 2 * F) - f.narrow(axis, F + b, n - 2 * F))
        return d

    @staticmethod
    def damp(d, m, p, half):
        a, b = (p["ah"], p["bh"]) if half else (p["a"], p["b"])
        m = b * m + a * d
        return d + m, m

    def add(self, f, inc):
        return f + torch.nn.functional.pad(inc, [self.fpad] * 4)

    def step(self, s):
        vx, vz, sxx, szx, szz = s[:5]
        m, F = list(s[5:]), self.fpad
        vx_x, m[0] = self.damp(self.diff(vx, 2, False), m[0], self.px, False)
        vz_x, m[1] = self.damp(self.diff(vz, 2, True), m[1], self.px, True)
        vx_z, m[2] = self.damp(self.diff(vx, 1, True), m[2], self.pz, True)
        vz_z, m[3] = self.damp(self.diff(vz, 1, False), m[3], self.pz, False)
        tr = self.lam * (vx_x + vz_z)
        szx = self.add(szx, DT * self.muzx * (vz_x + vx_z))
        sxx = self.add(sxx, DT * (tr + 2.0 * self.mu * vx_x))
        szz = self.add(szz, DT * (tr + 2.0 * self.mu * vz_z))
        if self.fsurf:  # stress-free surface row, images above it
            lam, mu = self.lam[0], self.mu[0]
            row = torch.nn.functional.pad(4.0 * DT * vx_x[:, :1] * (lam * mu + mu * mu) / (lam + 2.0 * mu), [F, F])
            sxx = torch.cat([sxx[:, :F], row, sxx[:, F + 1:]], 1)
            images = [-f[:, F + 1:2 * F + 1].flip(1) for f in (szx, szz)]
            zero = torch.zeros_like(row)
            szx = torch.cat([images[0], zero, szx[:, F + 1:]], 1)
            szz = torch.cat([images[1], zero, szz[:, F + 1:]], 1)
        sxx_x, m[4] = self.damp(self.diff(sxx, 2, True), m[4], self.px, False)
        szx_x, m[5] = self.damp(self.diff(szx, 2, False), m[5], self.px, True)
        szz_z, m[6] = self.damp(self.diff(szz, 1, True), m[6], self.pz, False)
        szx_z, m[7] = self.damp(self.diff(szx, 1, False), m[7], self.pz, True)
        vx = self.add(vx, DT * self.bx * (sxx_x + szx_z))
        vz = self.add(vz, DT * self.bz * (szx_x + szz_z))
        return [vx, vz, sxx, szx, szz, *m]


def _places(c, m):
    """Flat cells of the sources and of the receivers in the padded grid."""
    _, ppad, ztop = _padding(c, m["order"])
    nxt = m["nx"] + 2 * ppad
    return (torch.tensor((m["sz"] + ztop) * nxt + m["sx"] + ppad, dtype=torch.long),
            torch.tensor((m["rz"] + ztop) * nxt + m["rx"] + ppad, dtype=torch.long))


def _record(c, m, keep=False):
    """Traces [shot][rec][nt], final state and (keep) the fields before every sampled step; some shots at a time."""
    dev, nt, k = _device(), m["nt"], c["sample"]
    earth = [torch.from_numpy(a).to(dev) for a in m["earth"]]
    sch = _Scheme(c, m, earth)
    src, rec = (t.to(dev) for t in _places(c, m))
    sig = torch.from_numpy(m["sig"]).to(dev)
    per = sch.nzt * sch.nxt * 8 * (5 * (1 + (nt - 1) // k) if keep else 60)
    group = max(1, min(m["shots"], int(40e9 // per)))
    for b0 in range(0, m["shots"], group):
        ids = torch.arange(b0, min(b0 + group, m["shots"]), device=dev)
        row = torch.arange(len(ids), device=dev)
        s, fields, traces = sch.start(len(ids)), [], []
        for it in range(nt):
            if keep and it % k == 0:
                fields.append(s[:5])
            s = sch.step(s)
            v = s[1].reshape(len(ids), -1)
            v[row, src[ids]] += sig[it]
            traces.append(v[:, rec])
        yield sch, ids, torch.stack(traces, 2), s, fields


def _correlate(c, m):
    """Traces, misfits, per-shot gradients and the final states of the stored or checkpointed gradient."""
    dev, nt, k = _device(), m["nt"], c["sample"]
    nrec = len(m["rx"])
    obs = torch.from_numpy(m["obs"]).to(dev).reshape(m["shots"], nrec, nt)
    _, rec = (t.to(dev) for t in _places(c, m))
    recs, mis, grads, last = [], [], [], None
    for sch, ids, traces, fwd, fields in _record(c, m, keep=True):
        n, F = len(ids), sch.fpad
        res = traces - obs[ids]
        recs.append(traces)
        mis.append(0.5 * DT * res.square().sum((1, 2)))
        z1 = F if c["fsurf"] else 0
        win = (slice(None), slice(z1, sch.nzt, k), slice(0, sch.nxt, k))
        lam, mu = (torch.from_numpy(a).to(dev)[win[1:]] for a in m["earth"][:2])
        shape = (n, 1 + (sch.nzt - z1) // k, 1 + sch.nxt // k)
        g = [torch.zeros(shape, dtype=torch.float64, device=dev) for _ in range(3)]
        at = (slice(None), slice(0, lam.shape[0]), slice(0, lam.shape[1]))
        s = sch.start(n)
        ux = torch.zeros_like(s[0])
        uz = torch.zeros_like(s[0])
        inner = (slice(None), *sch.inner)
        for it in range(nt - 1, -1, -1):
            ux[inner] += DT * s[0][inner]
            uz[inner] += DT * s[1][inner]
            if it % k == 0:
                fvx, fvz, fxx, fzx, fzz = (f[win] for f in fields.pop())
                sxx, szx, szz = (f[win] for f in s[2:5])
                s1 = (fxx + fzz) * (sxx + szz) * 0.25 / (lam + mu) ** 2
                s2 = (fxx - fzz) * (sxx - szz) / mu ** 2
                g[0][at] += k * DT * s1
                g[1][at] += k * DT * (fzx * szx / mu ** 2 + s1 + s2)
                g[2][at] -= k * DT * (ux[win] * fvx + uz[win] * fvz) / DT
            s = sch.step(s)
            s[1].reshape(n, -1).index_add_(1, rec, res[:, :, it])
        grads.append(g)
        last = (fwd, s)
    return torch.cat(recs), torch.cat(mis), [torch.cat([g[q] for g in grads]) for q in range(3)], last


def _differentiate(c, m):
    """Misfit and its derivative with respect to lam, mu, rho, through the steps."""
    from torch.utils.checkpoint import checkpoint
    dev, nt = _device(), m["nt"]
    earth = [torch.from_numpy(a).to(dev).requires_grad_() for a in m["earth"]]
    src, rec = (t.to(dev) for t in _places(c, m))
    n, nrec = m["shots"], len(m["rx"])
    obs = torch.from_numpy(m["obs"]).to(dev).reshape(n, nrec, nt)
    sch = _Scheme(c, m, earth)
    row = torch.arange(n, device=dev)
    s, j = sch.start(n), 0.0

    def step(src_value, *s):
        s = sch.step(s)
        v = s[1].reshape(n, -1).index_put((row, src), src_value, accumulate=True)
        s[1] = v.reshape(s[1].shape)
        return tuple(s)

    for it in range(nt):
        value = torch.full((n,), float(m["sig"][it]), dtype=torch.float64, device=dev)
        s = checkpoint(step, value, *s, use_reentrant=False)
        j = j + 0.5 * DT * (s[1].reshape(n, -1)[:, rec] - obs[:, :, it]).square().sum()
    grads = list(torch.autograd.grad(j, earth))
    if c["fsurf"]:  # the gradient's window starts at the surface row
        for g in grads:
            g[:sch.fpad] = 0.0
    return j.detach(), grads


def exact(case, seed):
    cells = sum((nx + 2 * case["npml"]) * (nz + 2 * case["npml"]) * nt for nx, nz, _, nt, _ in _models(case))
    steps = cells * (1 if case["kind"] == "uneven" else case["shots"])
    if steps > 9e9 or (not torch.cuda.is_available() and steps > 2e7):
        return None  # longer than some 20 seconds
    ins = _inputs(case, seed)
    m, kind = ins[0], case["kind"]
    cpu = lambda t: t.cpu().numpy()  # noqa: E731
    if kind == "exact":
        j, g = _differentiate(case, m)
        return {"misfit": cpu(j), "grad": [cpu(t) for t in g]}
    if kind in ("forward", "misfit"):
        rec = torch.cat([t for _, _, t, _, _ in _record(case, m)])
        if kind == "forward":
            return {"rec": cpu(rec.reshape(-1, m["nt"]))}
        res = rec - torch.from_numpy(m["obs"]).to(rec.device).reshape(rec.shape)
        return {"misfit": cpu(0.5 * DT * res.square().sum((1, 2)))}
    if kind == "uneven":
        out = [_correlate(case, q) for q in ins]
        return {"misfit": np.array([float(o[1][0]) for o in out]),
                "grad": [[cpu(g[0, :q["earth"][0].shape[0], :q["earth"][0].shape[1]]) for g in o[2]]
                         for o, q in zip(out, ins)]}
    rec, mis, g, (fwd, adj) = _correlate(case, m)
    rec = cpu(rec.reshape(-1, m["nt"]))
    if kind == "reference":
        return {"rec": rec, "grad": [cpu(t[0]) for t in g], "forward": [cpu(t[0]) for t in fwd[:5]],
                "adjoint": [cpu(t[0]) for t in adj[:5]]}
    if kind == "stored":
        return {"rec": rec, "misfit": cpu(mis), "grad": [cpu(t) for t in g]}
    return {"misfit": cpu(mis), "grad": [cpu(t.sum(0)) for t in g]}
