"""The workloads this engine is timed on, as a user's program calls them.

Five kinds of work, each through the public binding (clmd.py, and the C
functions it binds):

  run    one system: the main loop for some steps, then the state back on the
         host (the drop-in; the mixed-precision NVT system);
  calls  one system driven call by call, as the Fortran host's loop does;
  frame  one stored configuration analysed: upload, list, forces, clusters,
         results back (restart and post-processing);
  ens    an ensemble of replicas advanced by windows, its state back on the
         host;
  admit  requests taken in, run and retired, as the served loop does between
         its rounds (its rounds themselves are sized by the clock, so that
         their results are not a function of the inputs).

Sizes, densities and temperatures are those of the tests, the decks and the
benchmark: 1,000 to 2,097,152 atoms in one system, 100 to 50,000 atoms in a
replica, rho* 0.01-0.05, T* 0.65-0.85, analysis every 50 or 100 steps.
"""
import ctypes as C
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                                "fortran-cluster-md_b200"))
import clmd  # noqa: E402

RC, RSKIN, ATSKIN, DT, NBTIM = 2.5, 2.8, 1.5, 0.005, 10
RMIN = 0.9
XV = ("x", "y", "z", "vx", "vy", "vz")
XVA = XV + ("ax", "ay", "az")


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # the smallest system of the configurations, ten analysis cycles per
        # read-out: latency of a step decides
        dict(name="run_1000_fp64_verlet", kind="run", n=1000, rho=0.01, temp=0.7, mixed=False,
             nose=False, twf=False, every=100, steps=1000),
        # a deck-sized system under Nose-Hoover (the reference's limit is 6000
        # atoms), an odd size
        dict(name="run_5921_fp64_nose", kind="run", n=5921, rho=0.03, temp=0.75, mixed=False,
             nose=True, twf=False, every=100, steps=200),
        # the FP64 drop-in workload
        dict(name="run_262144_fp64_verlet", kind="run", n=262144, rho=0.02, temp=0.7, mixed=False,
             nose=False, twf=False, every=100, steps=100),
        # the mixed-precision NVT workload, ten Wolde-Frenkel clusters
        dict(name="run_2097152_mixed_nose", kind="run", n=2097152, rho=0.05, temp=0.75, mixed=True,
             nose=True, twf=True, every=50, steps=50),
        # a Fortran host's loop over a small deck: velocity scaling and one
        # integrator call per step, an analysis every tenth
        dict(name="calls_2011_fp64_scaling", kind="calls", n=2011, rho=0.02, temp=0.7, every=10,
             steps=20),
        # a stored configuration with liquid droplets, ten Wolde-Frenkel
        dict(name="frame_30011_twf", kind="frame", n=30011, rho=0.05, temp=0.75, mixed=False,
             twf=True, drops=30),
        # a large stored vapour, Stillinger clusters
        dict(name="frame_1000003_stillinger", kind="frame", n=1000003, rho=0.02, temp=0.7,
             mixed=False, twf=False, drops=40),
        # the batched nucleation ensemble, states streamed to and from the host
        dict(name="ens_4096_mixed_nose_io", kind="ens", reps=4096, lo=200, hi=8000, rlo=0.01,
             rhi=0.05, tlo=0.65, thi=0.85, mixed=True, nose=True, windows=1, io=True, csover=51),
        # a few small replicas: one analysis window after another, latency
        dict(name="ens_61_small_mixed_nose", kind="ens", reps=61, lo=100, hi=1000, rlo=0.01,
             rhi=0.05, tlo=0.65, thi=0.85, mixed=True, nose=True, windows=2, io=False, csover=0),
        # an all-FP64 ensemble
        dict(name="ens_500_fp64_nose", kind="ens", reps=500, lo=200, hi=4000, rlo=0.01, rhi=0.05,
             tlo=0.65, thi=0.85, mixed=False, nose=True, windows=1, io=False, csover=51),
        # the largest replicas of the served workload
        dict(name="ens_9_large_mixed_nose", kind="ens", reps=9, lo=9000, hi=50000, rlo=0.01,
             rhi=0.05, tlo=0.65, thi=0.85, mixed=True, nose=True, windows=1, io=False, csover=101),
        # short requests: admitted, run, read out and removed
        dict(name="admit_64_mixed_nose", kind="admit", reps=64, lo=100, hi=20000, rlo=0.01,
             rhi=0.05, tlo=0.65, thi=0.85, mixed=True, nose=True, windows=2, io=False, csover=101),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["run", "run", "run", "calls", "frame", "ens", "ens", "ens", "admit"])
    rho = round(rng.uniform(0.01, 0.05), 4)
    temp = round(rng.uniform(0.65, 0.85), 3)
    if kind == "run":
        n = _log(rng, 1000, 2000000)
        every = rng.choice([50, 100])
        mixed = rng.random() < 0.5
        # FP32 pair terms and FP64 ones part ways within a few hundred steps
        cycles = 1 if mixed else max(1, min(10, int(2.0e7 / (n * every))))
        return dict(kind="run", n=n, rho=rho, temp=temp, mixed=mixed, nose=rng.random() < 0.5,
                    twf=rng.random() < 0.5, every=every, steps=every * cycles)
    if kind == "calls":
        return dict(kind="calls", n=_log(rng, 500, 6000), rho=rho, temp=temp, every=10, steps=20)
    if kind == "frame":
        n = _log(rng, 2000, 1500000)
        return dict(kind="frame", n=n, rho=rho, temp=temp, mixed=rng.random() < 0.5,
                    twf=rng.random() < 0.5, drops=min(40, n // 1000))
    if kind == "ens":
        if rng.random() < 0.25:  # large replicas
            reps, lo, hi = rng.randrange(1, 24), 9000, 50000
        else:
            lo = _log(rng, 100, 1000)
            hi = _log(rng, 2 * lo, 9000)
            reps = _log(rng, 16, 2048)
        return dict(kind="ens", reps=reps, lo=lo, hi=hi, rlo=0.01, rhi=0.05, tlo=0.65, thi=0.85,
                    mixed=rng.random() < 0.7, nose=rng.random() < 0.7, windows=1,
                    io=rng.random() < 0.4, csover=rng.choice([0, 51, 101]))
    return dict(kind="admit", reps=rng.randrange(1, 96), lo=100, hi=_log(rng, 1000, 20000),
                rlo=0.01, rhi=0.05, tlo=0.65, thi=0.85, mixed=rng.random() < 0.7, nose=True,
                windows=rng.choice([1, 2, 3]), io=False, csover=101)


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _vapour(rng, n, box):
    """n points in a cubic box, every pair at least RMIN apart: distinct cells
    of a grid, each point uniform in the part of its cell that keeps the
    distance to the neighbour cells."""
    m = int(box / 1.8)
    g = box / m
    cell = rng.permutation(m * m * m)[:n]
    at = np.stack([cell % m, cell // m % m, cell // (m * m)], 1)
    return at * g + rng.uniform(0.0, g - RMIN, (n, 3)) + 0.5 * RMIN


def _with_drops(rng, n, box, drops, radius=3.4, spacing=1.1):
    """A vapour with `drops` liquid droplets: cubic blobs of `spacing` in
    spheres that hold no vapour."""
    g = np.arange(-radius, radius + 1e-9, spacing)
    blob = np.stack([a.ravel() for a in np.meshgrid(g, g, g, indexing="ij")], 1)
    blob = blob[np.linalg.norm(blob, axis=1) <= radius]
    centres = np.zeros((0, 3))
    while len(centres) < drops:
        c = rng.uniform(0, box, 3)
        d = np.abs(centres - c)
        if (np.linalg.norm(np.minimum(d, box - d), axis=1) > 2 * radius + 3).all():
            centres = np.vstack([centres, c])
    gas = _vapour(rng, n, box)
    for c in centres:
        near = np.flatnonzero(np.abs(np.abs(gas[:, 0] - c[0]) - 0.5 * box) > 0.5 * box - 5.0)
        d = np.abs(gas[near] - c)
        d = np.linalg.norm(np.minimum(d, box - d), axis=1)
        gas = np.delete(gas, near[d <= radius + RMIN], 0)
    # a droplet holds more atoms than the vapour that made room for it
    return np.vstack([(blob + c) % box for c in centres] + [gas])[:n]


def _start(rng, n, box, temp, drops=0):
    pos = _with_drops(rng, n, box, drops) if drops else _vapour(rng, n, box)
    return [np.ascontiguousarray(pos[:, k]) for k in range(3)] + \
        [rng.normal(0.0, math.sqrt(temp), n) for _ in range(3)]


def _one_system(case, seed):
    n = case["n"]
    return _start(np.random.default_rng(seed), n, (n / case["rho"]) ** (1.0 / 3.0), case["temp"],
                  case.get("drops", 0))


def _mix(case):
    """(natom, box, temperature) of each replica: sizes log-uniform between
    lo and hi, densities and temperatures uniform, at the midpoints of equal
    shares of each range, in a shuffled order.  A property of the case: the
    seed makes the positions and velocities."""
    count = case["reps"]
    rng = np.random.default_rng(count)
    at = lambda: (rng.permutation(count) + 0.5) / count  # noqa: E731
    ns = np.exp(math.log(case["lo"]) + at() * math.log(case["hi"] / case["lo"])).astype(int)
    rhos = case["rlo"] + at() * (case["rhi"] - case["rlo"])
    temps = case["tlo"] + at() * (case["thi"] - case["tlo"])
    return [(n, (n / rho) ** (1.0 / 3.0), temp) for n, rho, temp in
            zip(ns.tolist(), rhos.tolist(), temps.tolist())]


def _replicas(case, seed):
    """(natom, box, temperature, x..vz) of each replica."""
    rng = np.random.default_rng(seed)
    return [(n, box, temp, _start(rng, n, box, temp)) for n, box, temp in _mix(case)]


# ---------------------------------------------------------------------------
# what a program has in hand, and one pass
# ---------------------------------------------------------------------------
def _config(case):
    scaled = case["kind"] == "calls"
    cfg = clmd.lj_config(
        case["n"], case["rho"], case["temp"], rc=RC, rskin=RSKIN, atskin=ATSKIN, dt=DT,
        nbtim=NBTIM, ftcsi=case.get("every", 100),
        integrator=clmd.INT_NOSE if case.get("nose") else clmd.INT_VERLET,
        ethst="X" if scaled else "N" if case.get("nose") else "-",
        clustering=clmd.CLU_FRENKEL if case.get("twf") else clmd.CLU_STILLINGER,
        precision=clmd.PREC_MIXED if case.get("mixed") else clmd.PREC_FP64)
    if scaled:
        cfg.apth = b"X" + b"-" * (clmd.MXSORTS - 1)
    return cfg


def _pinned(n, count):
    return {k: torch.empty(n, dtype=torch.float64).pin_memory().numpy() for k in XVA[:count]}


def _ptrs(bufs):
    return [clmd.ptr(a, C.c_double) for a in bufs.values()]


def _add(e, case, n, box, temp, arrs):
    return e.add(n, box, temp, *arrs, csover=case["csover"], budget=1 << 30,
                 ethst="N" if case["nose"] else "-")


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("run", "calls"):
        # main.f's start: momenta, list, accelerations, the thermostat's PSI
        cfg = _config(case)
        s = clmd.System(cfg)
        zero = np.zeros(case["n"])
        s.set_state(clmd.State(*_one_system(case, seed), zero, zero, zero),
                    scalars=clmd.scalars_init(cfg))
        s.stopdead(-1)
        s.neighbor(0)
        s.zero_acc()
        s.accatom()
        if case.get("nose"):
            q = s.scalars()
            q.psi = (2.0 * q.ekin - 3.0 * cfg.natom * clmd.CIKB * cfg.att) / cfg.Q
            s.set_scalars(q)
        bufs = _pinned(case["n"], 9)
        return dict(case=case, sys=s, step=0, bufs=bufs, ptrs=_ptrs(bufs))
    if kind == "frame":
        s = clmd.System(_config(case))
        bufs = _pinned(case["n"], 9)
        for k, a in zip(XV, _one_system(case, seed)):
            bufs[k][:] = a
        view, out = clmd.ClusterView(), {}
        for name, dt, size in clmd.CLUSTER_FIELDS:
            t = torch.empty(case["n"] + (size == "N1"),
                            dtype=torch.int32 if dt == np.int32 else torch.float64)
            out[name] = t.pin_memory().numpy()
            setattr(view, name, clmd.ptr(out[name], C.c_int32 if dt == np.int32 else C.c_double))
        return dict(case=case, sys=s, bufs=bufs, ptrs=_ptrs(bufs), view=view, clusters=out)
    # ens, admit
    reps = _replicas(case, seed)
    total = sum(r[0] for r in reps)
    e = clmd.Ensemble(clmd.ens_config(
        total, len(reps), precision=clmd.PREC_MIXED if case["mixed"] else clmd.PREC_FP64,
        integrator=clmd.INT_NOSE if case["nose"] else clmd.INT_VERLET, ftcsi=100, rc=RC,
        rskin=RSKIN, atskin=ATSKIN, dt=DT, nbtim=NBTIM))
    if kind == "admit":
        bufs = _pinned(total, 9)
        labels = torch.empty(total, dtype=torch.int32).pin_memory().numpy()
        at = np.concatenate([[0], np.cumsum([r[0] for r in reps])])
        ptrs = [[clmd.ptr(b[i:j], C.c_double) for b in bufs.values()] +
                [clmd.ptr(labels[i:j], C.c_int32)] for i, j in zip(at[:-1], at[1:])]
        return dict(case=case, ens=e, reps=reps, bufs=bufs, labels=labels, ptrs=ptrs)
    bufs, at = _pinned(total, 6), 0
    for n, box, temp, arrs in reps:
        _add(e, case, n, box, temp, arrs)
        for k, a in zip(XV, arrs):
            bufs[k][at:at + n] = a
        at += n
    return dict(case=case, ens=e, bufs=bufs, ptrs=_ptrs(bufs))


def _scalars(q):
    f = ("ekin", "epot", "psi", "s", "atrskin", "virial")
    i = ("npairs_half", "nrebuild", "maxcs", "cstep", "status")
    return {k: float(getattr(q, k)) for k in f}, {k: int(getattr(q, k)) for k in i}


def _results(got, energies=True):
    col = lambda k: np.array([getattr(got[r], k) for r in sorted(got)])  # noqa: E731
    out = {k: col(k) for k in ("step", "status", "done", "maxcs")}
    out["floats"] = {k: col(k) for k in ("ekin", "epot", "psi", "s")} if energies else None
    return out


def run(state):
    case, kind = state["case"], state["case"]["kind"]
    if kind in ("run", "calls"):
        s, step = state["sys"], state["step"]
        if kind == "run":
            _, state["step"] = s.run(step, case["steps"])
        else:
            for i in range(step, step + case["steps"]):
                if i % case["every"] == 0:
                    s.stoddard(i)
                s.thermostat(i)
                s.integrator(i)
            state["step"] = step + case["steps"]
        q = clmd.Scalars()
        s.lib.clmd_get_state(s.h, *state["ptrs"], C.byref(q))
        f, i = _scalars(q)
        return dict(state["bufs"], floats=f, ints=i, step=state["step"])
    if kind == "frame":
        s = state["sys"]
        null = [None] * 3
        s.lib.clmd_set_state(s.h, *state["ptrs"][:6], *null, None, None)
        s.neighbor(0)
        s.zero_acc()
        s.accatom()
        s.stoddard(0)
        q = clmd.Scalars()
        s.lib.clmd_get_state(s.h, *([None] * 6), *state["ptrs"][6:], C.byref(q))
        s.lib.clmd_get_clusters(s.h, C.byref(state["view"]))
        return dict({k: state["bufs"][k] for k in XVA[6:]}, clusters=state["clusters"],
                    epot=float(q.epot), virial=float(q.virial), pairs=int(q.npairs_half))
    e = state["ens"]
    if kind == "admit":
        slots = [_add(e, case, *r) for r in state["reps"]]
        e.step(case["windows"])
        got = e.results()
        for slot, ptrs in zip(slots, state["ptrs"]):
            e.lib.clmd_ens_get_state(e.h, slot, *ptrs)
            e.remove(slot)
        return dict(state["bufs"], cl=state["labels"], **_results(got))
    if case["io"]:
        e.step_io(case["windows"], state["ptrs"])
        return dict(state["bufs"], **_results(e.poll(), False))
    e.step(case["windows"])
    e.lib.clmd_ens_download(e.h, *state["ptrs"])
    return dict(state["bufs"], **_results(e.results()))


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def _step_flops(n, rho, steps):
    """Per atom and step: half the pairs within the list radius, about 40
    operations each, and about 60 for the integration."""
    return steps * n * (60.0 + 40.0 * 0.5 * rho * 4.18879 * RSKIN ** 3)


def work(case):
    kind = case["kind"]
    if kind in ("run", "calls"):
        return dict(bytes=144.0 * case["n"], flops=_step_flops(case["n"], case["rho"],
                                                               case["steps"]))
    if kind == "frame":
        ints = sum(4 if d == np.int32 else 8 for _, d, _ in clmd.CLUSTER_FIELDS)
        return dict(bytes=(48.0 + 24.0 + ints) * case["n"],
                    flops=_step_flops(case["n"], case["rho"], 1))
    lo, hi = case["lo"], case["hi"]
    mean = (hi - lo) / math.log(hi / lo) if hi > lo else lo  # of the log-uniform sizes
    rho = 0.5 * (case["rlo"] + case["rhi"])
    n = case["reps"] * mean
    return dict(bytes=(124.0 if kind == "admit" else 96.0) * n,
                flops=_step_flops(n, rho, 100 * case["windows"]))


# ---------------------------------------------------------------------------
# the same in 64 bits, with torch alone
# ---------------------------------------------------------------------------
class _Exact:
    """Systems of one species side by side, advanced together in FP64: atoms
    concatenated, system r holding atoms first[r] .. first[r + 1] in a cubic
    box, pairs from a list with a margin that a few steps cannot cross."""

    EVERY, MARGIN = 4, 0.6

    def __init__(self, parts, dev):
        """parts: (natom, box, temperature, x..vz) of each system."""
        f = dict(dtype=torch.float64, device=dev)
        self.dev, self.R = dev, len(parts)
        self.n = torch.tensor([p[0] for p in parts], device=dev)
        self.box = torch.tensor([p[1] for p in parts], **f)
        self.temp = torch.tensor([p[2] for p in parts], **f)
        self.rep = torch.repeat_interleave(torch.arange(self.R, device=dev), self.n)
        xv = [torch.from_numpy(np.concatenate([p[3][k] for p in parts])).to(dev) for k in range(6)]
        self.x, self.v = torch.stack(xv[:3], 1), torch.stack(xv[3:], 1)
        self.L = self.box[self.rep][:, None]
        self.pairs, self.age = None, 0
        zero = torch.zeros(self.R, **f)
        self.psi, self.s, self.dmms, self.dmmst = (zero.clone() for _ in range(4))
        self.skin = zero + RSKIN
        self.nkt3 = 3.0 * self.n * self.temp
        self.Q = self.n * self.temp * 0.25

    def sums(self, t):
        return torch.zeros(self.R, dtype=torch.float64, device=self.dev).index_add_(0, self.rep, t)

    def stopdead(self):
        for _ in range(10):
            for k in range(3):
                self.v[:, k] -= (self.sums(self.v[:, k]) / self.n)[self.rep]
            self.v *= torch.sqrt(self.nkt3 / self.sums((self.v ** 2).sum(1)))[self.rep][:, None]

    def wrap(self, which):
        w = torch.remainder(self.x, self.L)
        self.x = torch.where(which[self.rep][:, None], w, self.x)

    def find(self, radius):
        x = torch.remainder(self.x, self.L)
        nc = torch.floor(self.box / radius).long()
        if bool((nc < 3).any()):
            raise ValueError("box too small for the cell search")
        base = torch.cumsum(nc ** 3, 0) - nc ** 3
        m = nc[self.rep]
        c = torch.minimum((x / self.L * m[:, None]).long(), m[:, None] - 1)
        cell = base[self.rep] + (c[:, 2] * m + c[:, 1]) * m + c[:, 0]
        order = torch.argsort(cell)
        x, c, m, cell, L = x[order], c[order], m[order], cell[order], self.L[order]
        b = base[self.rep][order]
        count = torch.bincount(cell, minlength=int((nc ** 3).sum()))
        start = torch.cumsum(count, 0) - count
        ids = torch.arange(len(x), device=self.dev)
        got = []
        for dz in (-1, 0, 1):
            for dy in (-1, 0, 1):
                for dx in (-1, 0, 1):
                    if (dz, dy, dx) < (0, 0, 0):
                        continue
                    d = torch.tensor([dx, dy, dz], device=self.dev)
                    q = torch.remainder(c + d, m[:, None])
                    other = b + (q[:, 2] * m + q[:, 1]) * m + q[:, 0]
                    k = count[other]
                    i = torch.repeat_interleave(ids, k)
                    j = start[other][i] + torch.arange(len(i), device=self.dev) - \
                        (torch.cumsum(k, 0) - k)[i]
                    r = x[i] - x[j]
                    r -= L[i] * torch.round(r / L[i])
                    ok = (r * r).sum(1) <= radius * radius
                    if (dz, dy, dx) == (0, 0, 0):
                        ok &= j > i
                    got.append((order[i[ok]], order[j[ok]]))
        self.pairs = torch.cat([p[0] for p in got]), torch.cat([p[1] for p in got])
        self.age = 0

    def forces(self):
        """Accelerations; epot and virial of each system."""
        if self.pairs is None or self.age >= self.EVERY:
            self.find(RC + self.MARGIN)
        self.age += 1
        i, j = self.pairs
        r = self.x[i] - self.x[j]
        L = self.L[i]
        r -= L * torch.round(r / L)
        r2 = (r * r).sum(1)
        r6 = 1.0 / (r2 * r2 * r2)
        inside = r2 <= RC * RC
        f = torch.where(inside, 48.0 / r2 * r6 * (r6 - 0.5), 0.0)
        f3 = f[:, None] * r
        self.a = torch.zeros_like(self.x).index_add_(0, i, f3).index_add_(0, j, -f3)
        rep = self.rep[i]
        zero = torch.zeros(self.R, dtype=torch.float64, device=self.dev)
        self.epot = zero.index_add(0, rep, torch.where(inside, 4.0 * r6 * (r6 - 1.0), 0.0))
        self.virial = zero.index_add(0, rep, f * r2)

    def begin(self):
        self.stopdead()
        self.wrap(torch.ones(self.R, dtype=torch.bool, device=self.dev))
        self.forces()

    def step(self, step, nose, scaling=False):
        dth, dt2 = DT / 2, DT * DT / 2
        if scaling:
            self.v *= torch.sqrt(self.nkt3 / self.sums((self.v ** 2).sum(1)))[self.rep][:, None]
        drag = self.psi[self.rep][:, None] if nose else 0.0
        acc = self.a - drag * self.v
        dx = DT * self.v + dt2 * acc
        if nose:
            over = self.sums((self.v ** 2).sum(1)) - self.nkt3
            self.s = self.s + self.psi * DT + over * dt2 / self.Q
            self.psi = self.psi + over * dth / self.Q
        self.v = self.v + dth * acc
        self.x = self.x + dx
        # the adaptive list radius decides when positions are wrapped
        far = torch.zeros(self.R, dtype=torch.float64, device=self.dev).scatter_reduce_(
            0, self.rep, (dx * dx).sum(1), "amax")
        self.dmms = self.dmms + 2.2 * torch.sqrt(far)
        self.dmmst = self.dmmst + 1
        due = self.dmms > self.skin - RC - 2.0 * self.dmms / self.dmmst
        if bool(due.any()):
            self.wrap(due)
            if step > 0:
                new = torch.minimum(RC + (self.skin - RC) * NBTIM / self.dmmst, self.box / 2)
                self.skin = torch.where(due, new, self.skin)
            self.dmms = torch.where(due, 0.0, self.dmms)
            self.dmmst = torch.where(due, 0.0, self.dmmst)
        self.forces()
        w = self.v + dth * self.a
        total = self.sums((w * w).sum(1))
        if nose:  # v (1 + dth p) = w, p = psi + (sum v^2 - 3NkT) dth / Q
            p = self.psi.clone()
            for _ in range(8):
                c = 1.0 / (1.0 + dth * p)
                f = p - self.psi - (total * c * c - self.nkt3) * dth / self.Q
                p = p - f / (1.0 + 2.0 * total * dth * dth / self.Q * c ** 3)
            c = 1.0 / (1.0 + dth * p)
            self.psi, total = p, total * c * c
            w = w * c[self.rep][:, None]
        self.v, self.ekin = w, 0.5 * total


def exact(case, seed):
    kind = case["kind"]
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    many = kind in ("ens", "admit")
    parts = _replicas(case, seed) if many else \
        [(case["n"], (case["n"] / case["rho"]) ** (1.0 / 3.0), case["temp"],
          _one_system(case, seed))]
    steps = 100 * case["windows"] if many else case.get("steps", 1)
    if dev == "cpu" and sum(p[0] for p in parts) * steps > 5e6:
        return None
    e = _Exact(parts, dev)
    col = lambda t, k: t[:, k].cpu().numpy()  # noqa: E731
    if kind == "frame":
        e.MARGIN = 0.0
        e.wrap(torch.ones(1, dtype=torch.bool, device=dev))
        e.forces()
        return dict({k: col(e.a, n) for n, k in enumerate(XVA[6:])}, clusters=None,
                    epot=float(e.epot[0]), virial=float(e.virial[0]), pairs=None)
    e.begin()
    for i in range(steps):
        e.step(i, bool(case.get("nose")), scaling=kind == "calls")
    out = {k: col(e.x if n < 3 else e.v, n % 3) for n, k in enumerate(XV)}
    if kind != "ens":
        for n, k in enumerate(XVA[6:]):
            out[k] = col(e.a, n)
    if many:
        out["floats"] = None if case["io"] else {k: getattr(e, k).cpu().numpy() for k in
                                                 ("ekin", "epot", "psi", "s")}
        return dict(out, cl=None, step=None, status=None, done=None, maxcs=None)
    names = ("ekin", "epot", "psi", "s", "virial")
    return dict(out, floats=dict({k: float(getattr(e, k)[0]) for k in names},
                                 atrskin=float(e.skin[0])), ints=None, step=None)
