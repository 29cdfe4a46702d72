"""The work that users have this framework do, as cases to time and to compare.

Every case is one pass through the public entry points, from a state on the
GPU (or, for the job engine, on the host) to the results a program reads back:

``run``     one system through the fused loop, as simulation_md of the
            reference: upload, setup (cells, list, forces), `steps`
            iterations, records and the final state.  `steps` 0 is the start
            of a run alone: the forces and energies of a given configuration.
``calls``   the drop-in form: a host program that calls the reference's
            subroutines one by one, each iteration (md_advance_vv).
``melt``    a bead-spring polymer melt, or a Soddemann solution.
``batch``   independent replicas in one engine, as an ensemble study runs them.
``couette`` wall-driven channels in one engine (leap-frog, tethered and
            thermostatted walls, pressure tensor), as a serving loop gets them.
``noalloc`` forces into a caller's arrays, without any device allocation.

Sizes come from the benchmark configurations (2,048 WCA molecules, 1,048,576
LJ molecules, 262,144 FENE beads, replicas of 500-32,000, channels of
256-65,536) and the range between them, with odd and ragged boxes.

The FP32 form's trajectories come back as single-precision snapshots, the
precision of the reference's own vmd_temp.dcd; FP64 ones as they are.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

from flowmol_b200 import api, couette, lattice, polymer

WCA = 2.0 ** (1.0 / 6.0)
SKIN, DT = 0.3, 0.005
REC = ("iter", "simtime", "vsum", "mv2sum", "temperature", "kinenergy", "potenergy", "totenergy", "pressure",
       "virial")


def _run(name, nx, ny, nz, steps, **kw):
    """One LJ system of nx x ny x nz FCC units."""
    c = dict(kind="run", nx=nx, ny=ny, nz=nz, steps=steps, density=0.8442, temperature=0.722, rc=2.5, fp32=False,
             tplot=100, force_list=3, leapfrog=False, pressure=False, criterion=0, sort=0, shuffled=False)
    c.update(kw)
    return dict(name=name, **c) if name else c


def listed():
    return [
        # a host code that asks for forces of a small cluster every step: latency alone
        dict(name="noalloc_1k", kind="noalloc", nx=7, ny=6, nz=6, density=0.8, rc=2.5, fp32=False),
        # the smallest configuration of the benchmark set: short WCA runs of 2,048 molecules
        _run("wca_2k", 8, 8, 8, 100, rc=WCA, tplot=50),
        # below three cells per axis: all pairs
        _run("allpairs_500", 5, 5, 5, 60, force_list=0, fp32=True, tplot=20),
        # the reference's driver with its subroutines swapped for this library's
        dict(name="calls_31k", kind="calls", nx=20, ny=19, nz=21, steps=12, density=0.8442, temperature=0.722, rc=2.5,
             fp32=False),
        # a production run of a long-equilibrated liquid: numbering has nothing to do with place any
        # more; leap-frog, pressure tensor, frequent records
        _run("fluid_108k_lf", 30, 30, 30, 50, fp32=True, leapfrog=True, pressure=True, tplot=10, shuffled=True),
        # a ragged box in double precision, full-list force loop, thinner liquid
        _run("fluid_256k_f64", 39, 41, 40, 40, density=0.7, temperature=1.1, force_list=2, shuffled=True),
        # the headline configuration: 1M molecules, FP32 pair forces
        _run("fluid_1m", 64, 64, 64, 60, fp32=True),
        # restart of the 1M system in double precision: cells, list, forces and energies of its first step
        _run("start_1m_f64", 64, 64, 64, 0, shuffled=True),
        # the FENE melt of the benchmark set (262,144 beads)
        dict(name="melt_262k", kind="melt", chains=32768, beads=8, density=0.85, steps=50, fp32=True, solvent=False),
        # an ordinary polymer solution (Soddemann solvent) in double precision
        dict(name="solution_25k", kind="melt", chains=2091, beads=12, density=0.85, steps=40, fp32=False, solvent=True),
        # uneven LJ replicas in one engine
        dict(name="batch_40", kind="batch", jobs=40, smallest=500, largest=32000, steps=100, fp32=True),
        # Couette channels in one engine
        dict(name="couette_16", kind="couette", jobs=16, smallest=256, largest=40000, steps=120),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    """One more case: sizes over the logarithm of the declared range."""
    kind = rng.choice(["run", "run", "run", "run", "calls", "melt", "batch", "couette", "noalloc"])
    if kind == "noalloc":
        m = _log(rng, 5, 19)
        return dict(kind=kind, nx=round(m) + rng.randint(0, 1), ny=round(m), nz=round(m), density=rng.uniform(0.75, 0.9),
                    rc=rng.choice([WCA, 2.0, 2.5]) if m > 6 else WCA, fp32=rng.random() < 0.5)
    if kind == "calls":
        m = _log(rng, 10, 40)
        return dict(kind=kind, nx=round(m), ny=round(m) + rng.randint(0, 2), nz=round(m), steps=rng.randint(4, 12),
                    density=rng.uniform(0.7, 0.9), temperature=rng.uniform(0.7, 1.3), rc=2.5, fp32=rng.random() < 0.5)
    if kind == "melt":
        beads = rng.randint(4, 20)
        return dict(kind=kind, chains=round(_log(rng, 4000, 200000) / beads), beads=beads,
                    density=rng.uniform(0.8, 0.87), steps=rng.randint(10, 40), fp32=rng.random() < 0.5,
                    solvent=rng.random() < 0.4)
    if kind == "batch":
        return dict(kind=kind, jobs=rng.randint(2, 40), smallest=500, largest=round(_log(rng, 4000, 32000)),
                    steps=rng.randint(30, 80), fp32=rng.random() < 0.6)
    if kind == "couette":
        return dict(kind=kind, jobs=rng.randint(1, 16), smallest=256, largest=round(_log(rng, 2000, 40000)),
                    steps=rng.randint(30, 100))
    m = _log(rng, 9, 63)
    rc = rng.choice([2.5, 2.5, 2.5, WCA, 2.0, 3.0])
    big = m > 40
    return _run(None, round(m), round(m) + rng.randint(-1, 1), round(m) + rng.randint(-1, 1),
                rng.choice([0, 20, 40]) if big else rng.randint(20, 60), density=rng.uniform(0.6, 0.9),
                temperature=rng.uniform(0.7, 1.3), rc=rc, fp32=rng.random() < 0.5, tplot=rng.choice([10, 25, 100]),
                force_list=rng.choice([2, 3]), leapfrog=rng.random() < 0.25, pressure=rng.random() < 0.25,
                criterion=rng.choice([0, 0, 0, 2]), sort=rng.choice([0, 0, 0, 1, 2]), shuffled=rng.random() < 0.6)


# ---- inputs ---------------------------------------------------------------

def _fluid(c, seed):
    """A disordered FCC start on the GPU: (r, v, box), FP64."""
    g = torch.Generator("cuda").manual_seed(int(seed))
    nu = (c["nx"], c["ny"], c["nz"])
    box = lattice.global_domain(nu, c["density"])
    k = [torch.arange(n, dtype=torch.float64, device="cuda") for n in nu]
    cell = torch.stack(torch.meshgrid(k[2], k[0], k[1], indexing="ij"), -1).reshape(-1, 1, 3)[..., [1, 2, 0]]
    site = torch.tensor([[0, 0, 0], [.5, 0, .5], [0, .5, .5], [.5, .5, 0]], dtype=torch.float64, device="cuda")
    b = torch.tensor(box, device="cuda")
    r = ((cell + site + 0.25) * (b / torch.tensor(nu, dtype=torch.float64, device="cuda"))).reshape(-1, 3) - 0.5 * b
    r += (torch.rand(r.shape, generator=g, dtype=torch.float64, device="cuda") - 0.5) * 0.14
    v = torch.randn(r.shape, generator=g, dtype=torch.float64, device="cuda")
    v -= v.mean(0)
    v *= math.sqrt(c.get("temperature", 1.0) * 3 * len(r)) / v.norm()
    if c.get("shuffled"):
        p = torch.randperm(len(r), generator=g, device="cuda")
        r, v = r[p], v[p]
    return r.contiguous(), v.contiguous(), box


def _precision(c):
    return api.PRECISION_FP32 if c["fp32"] else api.PRECISION_FP64


def _sizes(c):
    """Job sizes, even in their logarithm, in an order of their own."""
    n = np.geomspace(c["smallest"], c["largest"], c["jobs"] + 1)[1:]
    return np.random.default_rng(c["jobs"]).permutation(n)


def _replicas(c, seed):
    fixed, rng = np.random.default_rng(c["largest"]), np.random.default_rng(seed)
    out = []
    for n in _sizes(c):
        m = max(2, round((n / 4.0) ** (1.0 / 3.0)))
        rho, temp = fixed.uniform(0.3, 0.9), rng.uniform(0.7, 1.5)
        r, v, box = lattice.lj_fluid([m, m, m], rho, temp, int(rng.integers(1 << 30)))
        pairs = 0 if min(np.floor(box / (2.5 + SKIN))) < 3 else 3
        out.append((api.make_job(len(r), box, 2.5, c["steps"], density=rho, force_list=pairs), r, v))
    return out


def _channels(c, seed):
    rng = np.random.default_rng(seed)
    out = []
    for n in _sizes(c):
        r, v, tag, rt, sv, box = couette.couette_job(couette.nunits_for(n), 0.8, 1.0, rng.uniform(0.5, 2.0),
                                                     int(rng.integers(1 << 30)))
        job = api.make_job(len(r), box, couette.WCA_RC, c["steps"], tplot=10, integration_algorithm=0, ensemble=6,
                           pressure_outflag=1, nthermo=2, thermostat_temperature=(1.0, 1.0), teth=(0.0, 5000.0, 5.0e6))
        out.append((job, r, v, tag, rt, sv))
    return out


_MELTS = {}


def _melt(c, seed):
    """Chain walks take seconds to grow at full size: one per size and
    composition, its velocities and a small displacement drawn from the seed."""
    key = (c["chains"], c["beads"], c["density"], c["solvent"])
    if key not in _MELTS:
        _MELTS.clear()
        _MELTS[key] = (polymer.fene_solution if c["solvent"] else polymer.fene_melt)(c["chains"], c["beads"], c["density"])
    r, _, chain, sub, _, bflag, box = _MELTS[key]
    g = torch.Generator("cuda").manual_seed(int(seed))
    r = torch.tensor(r, device="cuda") + (torch.rand(r.shape, generator=g, dtype=torch.float64, device="cuda") - 0.5) * 0.06
    v = torch.randn(r.shape, generator=g, dtype=torch.float64, device="cuda")
    v -= v.mean(0)
    v *= math.sqrt(3 * len(r)) / v.norm()
    return r, v, chain, sub, bflag, box


class State:
    """What a program holds between passes: inputs, the handle, its output arrays."""

    def __init__(self, **kw):
        self.__dict__.update(kw)


def prepare(case, seed):
    c, kind = case, case["kind"]
    if kind in ("batch", "couette"):
        jobs = _replicas(c, seed) if kind == "batch" else _channels(c, seed)
        mols = sum(j[0].np for j in jobs) + 1024
        eng = api.Engine(mols, 4 * mols, mols * 160, len(jobs), ticks_per_chunk=4096,
                         precision=_precision(c) if kind == "batch" else api.PRECISION_FP64)
        return State(case=c, jobs=jobs, eng=eng)
    if kind == "noalloc":
        r, _, box = _fluid(c, seed)
        L = api.lib()
        L.fm_compute_forces_noalloc.argtypes = [C.POINTER(api.FmParams), C.c_int32] + [C.c_void_p] * 5
        p = api.make_params(len(r), box, c["rc"], density=c["density"], precision=_precision(c))
        return State(case=c, p=p, L=L, r=r, a=torch.empty_like(r), pe=torch.empty_like(r[:, 0]),
                     vir=torch.empty_like(r[:, 0]))
    if kind == "melt":
        r, v, chain, sub, bflag, box = _melt(c, seed)
        p = api.make_params(len(r), box, WCA, (SKIN,) * 3, DT, 25, density=c["density"], precision=_precision(c),
                            potential_flag=1, k_c=30.0, R_0=1.5, solvent_flag=1 if c["solvent"] else 0)
        return State(case=c, s=api.MDSystem(p), r=r, v=v, mono=(chain, sub, bflag), out=[torch.empty_like(r) for _ in range(3)])
    r, v, box = _fluid(c, seed)
    p = api.make_params(len(r), box, c["rc"], (SKIN,) * 3, DT, c.get("tplot", 100), density=c["density"],
                        force_list=c.get("force_list", 3), rebuild_criteria=c.get("criterion", 0), precision=_precision(c),
                        integration_algorithm=0 if c.get("leapfrog") else 1)
    s = api.MDSystem(p)
    if c.get("pressure") or c.get("sort"):  # both are set once a state is there
        s.upload(r.cpu().numpy(), v.cpu().numpy())
    if c.get("pressure"):
        s.set_pressure_outflag(1)
    if c.get("sort"):
        s.set_sort(c["sort"], 1, 2)
    return State(case=c, s=s, r=r, v=v, out=[torch.empty_like(r) for _ in range(3)])


# ---- one pass -------------------------------------------------------------

def _upload(st):
    api.check(api.lib().fm_upload_state_device(st.s.h, st.s.n, C.c_void_p(st.r.data_ptr()), C.c_void_p(st.v.data_ptr())))


def _download(st, records):
    """Final r, v, a and the records, as the program keeps them."""
    api.check(api.lib().fm_download_state_device(st.s.h, *[C.c_void_p(x.data_ptr()) for x in st.out]))
    out = {k: x.float() if st.case["fp32"] else x for k, x in zip("rva", st.out)}
    out["records"] = np.array([[m[k] for k in REC] for m in records])
    return out


def run(state):
    st, c = state, state.case
    if c["kind"] in ("batch", "couette"):
        for j in st.jobs:
            st.eng.submit(*j)
        st.eng.run()
        res = sorted(st.eng.results(), key=lambda x: x["job_id"])
        kind = np.float32 if c.get("fp32") else np.float64
        out = [np.concatenate([np.asarray(x, kind) for x in st.eng.job_state(q["job_id"], j[0].np)])
               for q, j in zip(res, st.jobs)]
        last = np.array([[q["last"][k] for k in REC] for q in res], kind)
        return {"state": np.concatenate(out), "last": last, "ptensor": np.stack([q["ptensor"] for q in res]).astype(kind),
                "status": np.array([q["status"] for q in res])}
    if c["kind"] == "noalloc":
        rc = st.L.fm_compute_forces_noalloc(C.byref(st.p), len(st.r), st.r.data_ptr(), st.a.data_ptr(), st.pe.data_ptr(),
                                            st.vir.data_ptr(), None)
        if rc:
            raise RuntimeError("fm_compute_forces_noalloc: %d" % rc)
        return {"a": st.a, "pe": st.pe, "vir": st.vir}
    s = st.s
    _upload(st)
    if c["kind"] == "melt":
        s.upload_monomers(*st.mono)
    s.setup()
    if c["kind"] == "calls":
        for _ in range(c["steps"]):
            s.md_advance_vv()
        return _download(st, [s.evaluate_macroscopic_properties()])
    if c["steps"]:
        s.simulation_md(c["steps"])
    out = _download(st, s.records(64))
    if c.get("pressure"):
        out["ptensor"] = s.pressure_tensor(True)[0]
    if not c["steps"]:
        out["pe"], out["virial"] = s.per_molecule()
    return out


# ---- what a pass cannot do without -----------------------------------------

def _size(c):
    """(molecules, pairs inside the cutoff per molecule, force evaluations)."""
    if c["kind"] == "melt":
        return c["chains"] * c["beads"], 2 / 3 * math.pi * WCA ** 3 * c["density"] + 1, c["steps"] + 1
    n = 4 * c["nx"] * c["ny"] * c["nz"]
    return n, min(2 / 3 * math.pi * c["rc"] ** 3 * c["density"], (n - 1) / 2), c.get("steps", 0) + 1


def work(case):
    """Per force evaluation: r, v, a of every molecule read and written once
    (192 bytes; forces alone: 24 in, 40 out), and about 30 operations for each
    pair inside the cutoff, met once."""
    if case["kind"] in ("batch", "couette"):
        lo, hi = case["smallest"], case["largest"]  # sizes are uniform in their logarithm
        n = case["jobs"] * (hi - lo) / math.log(hi / lo)
        pairs = 2 / 3 * math.pi * (2.5 ** 3 * 0.6 if case["kind"] == "batch" else WCA ** 3 * 0.8)
        evals = case["steps"] + 1
    else:
        n, pairs, evals = _size(case)
    return {"bytes": n * (64.0 if case["kind"] == "noalloc" else 192.0 * evals), "flops": 30.0 * n * pairs * evals}


# ---- the same in plain FP64 -------------------------------------------------

def _pairs(r, box, reach):
    """(i, j), i < j or in another cell, of all pairs within `reach`."""
    n = len(r)
    nc = [int(b / reach) for b in box.tolist()]
    if min(nc) < 3:
        i, j = torch.triu_indices(n, n, 1, device=r.device)
        d = r[i] - r[j]
        d -= box * torch.round(d / box)
        k = (d * d).sum(1) < reach * reach
        return i[k], j[k]
    m = torch.tensor(nc, device=r.device)
    q = torch.remainder(torch.floor((r / box + 0.5) * m).long(), m)
    cell = (q[:, 2] * nc[1] + q[:, 1]) * nc[0] + q[:, 0]
    order = torch.argsort(cell)
    count = torch.bincount(cell, minlength=nc[0] * nc[1] * nc[2])
    first = torch.cumsum(count, 0) - count
    cap = int(count.max())
    table = torch.full((len(count), cap), n, device=r.device)
    table[cell[order], torch.arange(n, device=r.device) - first[cell[order]]] = order
    rp = torch.cat([r, torch.full((1, 3), float("nan"), dtype=r.dtype, device=r.device)])
    ids = torch.arange(len(count), device=r.device)
    x, y, z = ids % nc[0], ids // nc[0] % nc[1], ids // (nc[0] * nc[1])
    out_i, out_j = [], []
    step = max(1, 4_000_000 // (cap * cap))
    for s in range(14):  # the cell itself and the 13 that follow it
        dx, dy, dz = (s + 13) % 3 - 1, (s + 13) // 3 % 3 - 1, (s + 13) // 9 - 1
        other = ((z + dz) % nc[2] * nc[1] + (y + dy) % nc[1]) * nc[0] + (x + dx) % nc[0]
        for c0 in range(0, len(ids), step):
            a, b = table[c0:c0 + step], table[other[c0:c0 + step]]
            d = rp[a][:, :, None] - rp[b][:, None]
            d -= box * torch.round(d / box)
            near = (d * d).sum(-1) < reach * reach
            if s == 0:
                near &= a[:, :, None] < b[:, None]
            k = near.nonzero()
            out_i.append(a[k[:, 0], k[:, 1]])
            out_j.append(b[k[:, 0], k[:, 2]])
    return torch.cat(out_i), torch.cat(out_j)


class _Exact:
    """Truncated and shifted LJ, and FENE bonds, of one periodic system."""

    def __init__(self, r, box, rc, bonds=None):
        self.r, self.rc, self.bonds = r.clone(), rc, bonds
        self.box = torch.as_tensor(box, dtype=torch.float64, device=r.device)
        self.left = 0

    def _apart(self, i, j):
        d = self.r[i] - self.r[j]
        return d - self.box * torch.round(d / self.box)

    def forces(self, energies=False):
        n = len(self.r)
        if self.left == 0:  # pairs within 0.5 of the cutoff stay complete for 8 steps
            self.i, self.j = _pairs(self.r, self.box, self.rc + 0.5)
            self.left = 8
        self.left -= 1
        a = torch.zeros_like(self.r)
        pe, vir = torch.zeros_like(self.r[:, 0]), torch.zeros_like(self.r[:, 0])
        shift = 4 * (self.rc ** -12 - self.rc ** -6)
        for k in range(0, len(self.i), 8_000_000):
            i, j = self.i[k:k + 8_000_000], self.j[k:k + 8_000_000]
            d = self._apart(i, j)
            r2 = (d * d).sum(1)
            near = r2 < self.rc * self.rc
            i, j, d, r2 = i[near], j[near], d[near], r2[near]
            s3 = r2 ** -3
            f = 48 * (s3 * s3 - 0.5 * s3) / r2
            a.index_add_(0, i, f[:, None] * d)
            a.index_add_(0, j, -f[:, None] * d)
            if energies:
                for at in (i, j):
                    pe.index_add_(0, at, 4 * (s3 * s3 - s3) - shift)
                    vir.index_add_(0, at, f * r2)
        if self.bonds is not None:
            i, j = self.bonds
            d = self._apart(i, j)
            f = (-30.0 / (1 - (d * d).sum(1) / 2.25))[:, None] * d
            a.index_add_(0, i, f)
            a.index_add_(0, j, -f)
        return a, pe, vir


def exact(case, seed):
    """Forces, energies and short velocity-Verlet trajectories in plain torch.
    When a molecule is wrapped into the box hangs on the rebuild steps, so v
    and a stand for a trajectory here, not r."""
    c = case
    if c["kind"] == "noalloc":
        r, _, box = _fluid(c, seed)
        a, pe, vir = _Exact(r, box, c["rc"]).forces(True)
        return {"a": a, "pe": pe, "vir": vir}
    if c["kind"] in ("batch", "couette") or c.get("leapfrog") or c.get("solvent") or c.get("sort"):
        return None
    bonds = None
    if c["kind"] == "melt":
        r, v, chain, sub, _, box = _melt(c, seed)
        k = torch.arange(len(r), device="cuda").reshape(-1, c["beads"])
        bonds = (k[:, :-1].reshape(-1), k[:, 1:].reshape(-1))
    else:
        r, v, box = _fluid(c, seed)
    if len(r) * c["steps"] > 70_000_000:
        return None
    x, v = _Exact(r, box, c.get("rc", WCA), bonds), v.clone()
    a, pe, vir = x.forces(not c["steps"])
    for _ in range(c["steps"]):
        x.r += DT * v + 0.5 * DT * DT * a
        v += 0.5 * DT * a
        a, _, _ = x.forces()
        v += 0.5 * DT * a
    out = {"r": None if c["steps"] else x.r, "v": v, "a": a, "records": None}
    if c.get("pressure"):
        out["ptensor"] = None
    if not c["steps"]:
        out["pe"], out["virial"] = pe, vir
    return out
