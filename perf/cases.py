"""The measured cases: what a program that uses this framework has it do.

Five kinds of work, each through the entry point such a program calls:

  noalloc  sg_compute_forces_noalloc on device buffers: one force evaluation (cell sort, lists,
           forces) for a caller that owns the device memory, up to 16,384 atoms
  step     a snapshot of one or many systems loaded, its lists built, a block of time steps on
           device-resident state, then the new state read back (how trajectories are sampled)
  host     one step from host arrays (Simulation.step_from_host) and the state back: a host
           program that owns the state, the end-to-end form
  diff     energies, forces, or the force-matching loss of the fitted model over a set of frames,
           with the gradient with respect to its 66 parameters where it has one (one iteration
           of a fit)
  rdf      a radial-distribution sample of a system (stencil histogram and the 0-15 A extension)

Systems are the repository's workloads (surfacegrowthconsole_gb300.workloads): graphene sheets of
32 ux uy carbon atoms with metal clusters, and bulk fcc metals.  Atoms start displaced by a thermal
0.05 A (frozen sheet edges excepted, which a simulation never moves), as snapshots of a running
simulation are, not on the perfect lattice, where most forces cancel.
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

from surfacegrowthconsole_gb300 import MODE_MIXED, MODE_PLAIN, _lib, workloads
from surfacegrowthconsole_gb300.engine import (DIFF_NPARAM, DiffModel, Simulation, build_workload, diff_frame_params,
                                               diff_init_theta)

LENGTH_A = 1.42      # the framework's length unit in angstrom
JITTER = 0.05 / LENGTH_A
RDF_BINS, RDF_RANGE = 300, 15.0 / LENGTH_A
LAST = 10 ** 8       # step limits out of the way: the thermostat stays on, the shear drive off


# ------------------------------------------------------------------------------------------
# the cases
# ------------------------------------------------------------------------------------------
def listed():
    return [
        # the smallest call: one force evaluation of the 2,217-atom system under another
        # framework's memory manager; launches and latency
        {"name": "noalloc_small", "kind": "noalloc", "ux": 7, "uy": 9, "clusters": "201", "T": 300.0},
        # the same call near its size limit, a ragged size
        {"name": "noalloc_large", "kind": "noalloc", "ux": 19, "uy": 24, "clusters": "1291", "T": 700.0},
        # the small configuration (graphene + 201 Ni, 300 K), PLAIN drop-in form, lists by the
        # reference's rule: a desktop-size run, bound by the step's latency
        {"name": "step_small_plain", "kind": "step", "mode": "plain", "rebuild": False, "ux": 7, "uy": 9,
         "clusters": "201", "T": 300.0, "reps": 1, "steps": 10, "tuned": False},
        # the production configuration (40,000 C + 8 Ni clusters, 700 K, lists rebuilt every
        # step), MIXED form
        {"name": "step_production_mixed", "kind": "step", "mode": "mixed", "rebuild": True, "ux": 25, "uy": 50,
         "clusters": "868,627,440,545,702,823,906,635", "T": 700.0, "reps": 1, "steps": 10, "tuned": False},
        # one step of the same system from host arrays, PLAIN drop-in form
        {"name": "host_production_plain", "kind": "host", "mode": "plain", "rebuild": True, "ux": 25, "uy": 50,
         "clusters": "868,627,440,545,702,823,906,635", "T": 700.0, "reps": 1, "steps": 1, "tuned": False},
        # bulk Au, 24^3 unit cells (a configuration the reference published), PLAIN form
        {"name": "step_bulk_au_plain", "kind": "step", "mode": "plain", "rebuild": False, "bulk": 24, "material": 2,
         "T": 300.0, "reps": 1, "steps": 10, "tuned": False},
        # many uneven replicas advancing together (parameter sweeps): the throughput form, with
        # the launch shape autotuning reports for it
        {"name": "step_batched_mixed", "kind": "step", "mode": "mixed", "rebuild": False, "T": 0.0, "reps": 64,
         "steps": 10, "tuned": True},
        # one iteration of a fit to a few small frames
        {"name": "diff_fit_small", "kind": "diff", "what": "loss_grad", "ux": 7, "uy": 9, "clusters": "201",
         "T": 300.0, "frames": 4},
        # one iteration of the full fit: 64 frames of the 20,432-atom system
        {"name": "diff_fit_large", "kind": "diff", "what": "loss_grad", "ux": 24, "uy": 24, "clusters": "2000",
         "T": 700.0, "frames": 64},
        # energies and their gradient over a subset of the frames
        {"name": "diff_energy_grad", "kind": "diff", "what": "energy_grad", "ux": 24, "uy": 24, "clusters": "2000",
         "T": 700.0, "frames": 16},
        # forces of the fitted model on a validation set of odd-sized frames
        {"name": "diff_forces", "kind": "diff", "what": "forces", "ux": 11, "uy": 13, "clusters": "777",
         "T": 700.0, "frames": 24},
        # a radial-distribution sample of the production system
        {"name": "rdf_production", "kind": "rdf", "ux": 25, "uy": 50, "clusters": "868,627,440,545,702,823,906,635",
         "T": 700.0},
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _sheet(rng, cells_lo, cells_hi, umin=3):
    """A nearly square sheet of about so many 32-atom graphene units (log-uniform)."""
    cells = _logint(rng, cells_lo, cells_hi)
    ux = max(umin, int(round(math.sqrt(cells * 6 / (8 * math.cos(math.pi / 6))))) + rng.randint(-1, 1))
    return ux, max(umin, int(round(cells / ux)))


def draw(rng):
    """One more case of the same ranges."""
    kind = rng.choice(["noalloc", "step", "step", "host", "diff", "diff", "rdf"])
    T = float(rng.randint(300, 1500 if kind in ("step", "host") else 1000))
    if kind == "noalloc":
        ux, uy = _sheet(rng, 63, 440, 7)
        return {"kind": kind, "ux": ux, "uy": max(uy, 7), "clusters": str(_logint(rng, 50, 1600)), "T": T}
    if kind == "diff":
        ux, uy = _sheet(rng, 80, 576, 8)
        return {"kind": kind, "what": rng.choice(["loss_grad", "loss_grad", "energy_grad", "forces"]), "ux": ux,
                "uy": max(uy, 9), "clusters": str(_logint(rng, 50, 2000)), "T": T, "frames": _logint(rng, 1, 48)}
    if kind == "rdf":
        ux, uy = _sheet(rng, 120, 1250, 7)
        return {"kind": kind, "ux": ux, "uy": uy,
                "clusters": ",".join(str(_logint(rng, 50, 900)) for _ in range(rng.randint(1, 4))), "T": T}
    c = {"kind": kind, "mode": rng.choice(["plain", "mixed"]), "rebuild": rng.random() < 0.4, "T": T, "reps": 1,
         "steps": 10 if kind == "step" else 1, "tuned": False}
    form = rng.choice(["sheet", "sheet", "bulk", "batched"]) if kind == "step" else "sheet"
    if form == "bulk":
        c.update(bulk=_logint(rng, 6, 28), material=rng.randint(0, 5), T=300.0)
    elif form == "batched":
        c.update(T=0.0, reps=_logint(rng, 2, 48), tuned=rng.random() < 0.5)
    else:
        ux, uy = _sheet(rng, 30, 2500, 4)
        many = 1 if ux * uy < 300 else rng.randint(1, 8)
        c.update(ux=ux, uy=uy, clusters=",".join(str(_logint(rng, 50, 1000)) for _ in range(many)))
    return c


# ------------------------------------------------------------------------------------------
# inputs
# ------------------------------------------------------------------------------------------
def _thermal(p, r, rng):
    """r with a thermal displacement of every atom a simulation would have moved."""
    c30 = np.float32(math.cos(math.pi / 6.0))
    n = p.nMol
    x, y = r[:, 0], r[:, 1]
    half = np.float32(0.5)
    Lx, Ly = np.float32(p.region.x), np.float32(p.region.y)
    frozen = ~((x != half * (c30 - Lx)) & (x < half * (Lx - c30)) & (y != half * (Ly - np.float32(1))) &
               (y != half * (np.float32(1) - Ly)))
    frozen[:p.nMolMe] = False
    d = rng.normal(0, JITTER, size=(n, 3)).astype(np.float32)
    d[frozen] = 0
    out = r.copy()
    out[:, :3] += d
    out[:, 3] = 0
    return out


def _system(case, seed):
    """(parameter block, positions, velocities) of a one-system case."""
    rng = np.random.RandomState(seed % (1 << 31))
    if case.get("bulk"):
        p, r, v = workloads.bulk_metal(case["bulk"], case["T"], seed=seed % 100000 + 1, material=case["material"])
    else:
        p, r, v = build_workload(case["ux"], case["uy"], [int(s) for s in case["clusters"].split(",")], case["T"],
                                 seed, step_limit=LAST, step_avg=100, step_equil=0, step_cool=LAST, step_rdf=100,
                                 limit_rdf=10, step_diffuse=10, n_val_diffuse=100, n_buff_diffuse=10,
                                 limit_diffuse_av=5, delta_t=workloads.DT_1FS)
    return p, _thermal(p, r, rng), v


def _systems(case, seed):
    """The replicas of a step case: one system, or the uneven batch."""
    if case["reps"] == 1:
        return [_system(case, seed)]
    # the sizes and temperatures of the batched workload (one set, whatever the seed), the
    # cluster positions, displacements and velocities from the seed
    sizes, rng, out = np.random.RandomState(4), np.random.RandomState(seed % (1 << 31)), []
    for k in range(case["reps"]):
        cells = max(4, int(round(sizes.uniform(1000, 20000) / 32)))
        ux = max(2, int(round(math.sqrt(cells * 6 / (8 * math.cos(math.pi / 6))))))
        p, r, v = build_workload(ux, max(2, int(round(cells / ux))), [int(sizes.randint(50, 2001))],
                                 float(sizes.uniform(300, 1500)), (seed % 20000) * 1000 + k, step_limit=LAST,
                                 step_avg=100, step_equil=0, step_rdf=100, limit_rdf=10,
                                 delta_t=workloads.DT_1FS)
        out.append((p, _thermal(p, r, rng), v))
    return out


def _frames(case, seed):
    """Frame parameter block and the positions of all frames."""
    p, r, _ = build_workload(case["ux"], case["uy"], [int(s) for s in case["clusters"].split(",")], case["T"], seed,
                             step_limit=LAST, delta_t=workloads.DT_1FS)
    rng = np.random.RandomState(seed % (1 << 31))
    return diff_frame_params(p), [_thermal(p, r, rng) for _ in range(case["frames"])]


def _theta_ref(case, seed, q, n):
    """A guess of the parameters in mid-fit and reference forces (a few eV/A)."""
    rng = np.random.RandomState((seed + 1) % (1 << 31))
    theta = diff_init_theta(q) * (1 + 0.02 * rng.normal(size=DIFF_NPARAM))
    return theta, rng.normal(0, 1.0, size=(n, 3)).astype(np.float32)


_TUNED = {"metal_lanes": 4, "nebr_blocks_per_sm": 7, "nebr_item_atoms": 16, "carbon_blocks_per_sm": 16}


def prepare(case, seed):
    kind = case["kind"]
    if kind == "noalloc":
        p, r, _ = _system(case, seed)
        return {"kind": kind, "p": p, "pos": torch.from_numpy(r).cuda(),
                "acc": torch.zeros((p.nMol, 4), dtype=torch.float32, device="cuda")}
    if kind == "diff":
        q, frames = _frames(case, seed)
        theta, ref = _theta_ref(case, seed, q, q.nMol * case["frames"])
        model = DiffModel([q] * case["frames"], np.concatenate(frames))
        return {"kind": kind, "what": case["what"], "model": model, "theta": theta, "ref": ref}
    if kind == "rdf":
        p, r, v = _system(case, seed)
        sim = Simulation(p, mode=MODE_MIXED, rdf_ext_bins=RDF_BINS, rdf_ext_range=RDF_RANGE)
        sim.set_state(r, v, np.zeros((p.nMol, 3), np.float32))
        sim.build_lists()
        return {"kind": kind, "sim": sim}
    systems = _systems(case, seed)
    r, v = (np.ascontiguousarray(np.concatenate([s[k] for s in systems])) for k in (1, 2))
    a = np.zeros((len(r), 3), np.float32)
    shape = _TUNED if case["tuned"] else {}
    sim = Simulation([s[0] for s in systems], mode=MODE_MIXED if case["mode"] == "mixed" else MODE_PLAIN,
                     force_rebuild=case["rebuild"], **shape)
    return {"kind": kind, "sim": sim, "steps": case["steps"], "r": r, "v": v, "a": a,
            "build": kind == "step" and not case["rebuild"]}


# ------------------------------------------------------------------------------------------
# one pass
# ------------------------------------------------------------------------------------------
def _snapshot(sim, t):
    r, v, a = sim.get_state()
    # the energies of the record (per atom, replica 0) beside the whole state
    return {"r": r, "v": v, "a": a,
            "thermo": np.array([t.kinEnergy, t.potEnergy, t.totEnergy, t.vvSum, t.vvMax, t.uSum], np.float32)}


def run(s):
    kind = s["kind"]
    if kind == "step":
        sim = s["sim"]
        sim.set_state(s["r"], s["v"], s["a"])
        if s["build"]:  # otherwise the first step does
            sim.build_lists()
        return _snapshot(sim, sim.step_thermo(s["steps"]))
    if kind == "host":
        t = s["sim"].step_from_host(s["r"], s["v"], s["a"], nsteps=s["steps"])
        return _snapshot(s["sim"], t)
    if kind == "noalloc":
        pos, acc = s["pos"], s["acc"]
        _lib.check(_lib.lib().sg_compute_forces_noalloc(
            ctypes.byref(s["p"]), ctypes.c_void_p(pos.data_ptr()), ctypes.c_void_p(acc.data_ptr()),
            ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
        return {"pos": pos, "acc": acc}
    if kind == "rdf":
        sim = s["sim"]
        sim.reset_rdf()
        sim.eval_rdf()
        return {"hist": sim.rdf(0).astype(np.int64), "ext": sim.rdf_ext(0, RDF_BINS).astype(np.int64)}
    m = s["model"]
    if s["what"] == "loss_grad":
        loss, g = m.force_matching(s["theta"], s["ref"])
        return {"loss": np.array([loss], np.float32), "grad": g.astype(np.float32)}
    if s["what"] == "energy_grad":
        e, g = m.energy(s["theta"])
        return {"energy": e.astype(np.float32), "grad": g.astype(np.float32)}
    return {"forces": m.forces(s["theta"])}


# ------------------------------------------------------------------------------------------
# what a pass cannot do without
# ------------------------------------------------------------------------------------------
def _counts(case):
    """(carbon atoms, metal atoms) of one system (the mean one of a batch)."""
    if case.get("bulk"):
        return 0, 4 * case["bulk"] ** 3
    if case.get("reps", 1) > 1:
        return 10500, 1025
    return 32 * case["ux"] * case["uy"], sum(int(s) for s in case["clusters"].split(","))


def work(case):
    nc, nm = _counts(case)
    reps = case.get("reps", 1) * case.get("frames", 1)
    n = (nc + nm) * reps
    # flops of one evaluation: a metal atom has about 45 metal neighbours within the cutoff (a
    # density and a pair term, about 60 flops) and a few carbon ones, a carbon atom 9 angles of
    # about 60 flops
    forces = reps * (nm * 45 * 60 + nc * 9 * 60)
    kind = case["kind"]
    if kind == "noalloc":
        return {"bytes": n * (16 + 4 + 16), "flops": forces}
    if kind == "rdf":
        return {"bytes": n * 16 + 12 * RDF_BINS, "flops": nm * nm * 4}
    if kind == "diff":
        pairs = reps * nm * 45
        if case["what"] == "forces":
            return {"bytes": n * (16 + 12), "flops": pairs * 80}
        if case["what"] == "energy_grad":
            return {"bytes": n * 16 + 8 * DIFF_NPARAM, "flops": pairs * 100}
        return {"bytes": n * (16 + 12) + 8 * DIFF_NPARAM, "flops": pairs * 200}
    # the state (r, v, a) read and written once, whatever the number of steps
    return {"bytes": n * 80, "flops": case["steps"] * (forces + 60 * n)}


# ------------------------------------------------------------------------------------------
# the same in 64 bits
# ------------------------------------------------------------------------------------------
_MOST_ATOMS = 60000   # of one system: the pair search below is all against all


def _dev():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _wrap(d, L):
    """Minimum image, one box at most."""
    return d - L * ((d >= 0.5 * L).double() - (d < -0.5 * L).double())


class _Model64:
    """The model of one parameter block in 64 bits: EAM metal, Lennard-Jones metal-carbon over the
    neighbour list, graphene bonds over the first three close carbons in list order."""

    def __init__(self, p, r):
        self.p, self.n, self.m = p, p.nMol, p.nMolMe
        self.L = torch.tensor([p.region.x, p.region.y, p.region.z], dtype=torch.float64, device=_dev())
        self.cells = torch.tensor([p.cells.x, p.cells.y, p.cells.z], device=_dev())
        self.inv = torch.tensor([p.invWidth.x, p.invWidth.y, p.invWidth.z], dtype=torch.float64, device=_dev())
        self.I, self.K = self._near(r, math.sqrt(p.rrNebr) + 0.3)

    def _near(self, r, cut):
        """Pairs (i, k), both directions, that can come within the list radius in a few steps."""
        x, L = r.float(), self.L.float()
        I, K = [], []
        step = max(1, (1 << 26) // self.n)
        for b in range(0, self.n, step):
            d2 = 0
            for k in range(3):
                d = (x[b:b + step, None, k] - x[None, :, k]).abs_()
                d2 = d2 + torch.minimum(d, L[k] - d) ** 2
            i, k = (d2 < cut * cut).nonzero(as_tuple=True)
            i = i + b
            keep = i != k
            I.append(i[keep])
            K.append(k[keep])
        return torch.cat(I), torch.cat(K)

    def build(self, r):
        """The neighbour list in the framework's order: by stencil cell, then by atom index."""
        d = _wrap(r[self.I] - r[self.K], self.L)
        keep = (d * d).sum(1) < self.p.rrNebr
        I, K = self.I[keep], self.K[keep]
        c = ((r + 0.5 * self.L) * self.inv).long()
        o = (c[K] - c[I]) % self.cells            # 0, 1 or cells - 1 along each axis
        o = torch.where(o == self.cells - 1, torch.full_like(o, 2), o)
        o = o[:, 0] * 9 + o[:, 1] * 3 + o[:, 2]
        order = torch.argsort((I * 32 + o) * self.n + K)
        self.i, self.k = I[order], K[order]
        count = torch.bincount(self.i, minlength=self.n)
        first = torch.cumsum(count, 0) - count
        self.j = torch.arange(len(self.i), device=r.device) - first[self.i]

    def _three(self, sel):
        """Entries sel (a mask over the list): each atom's first three, as list indices, and how many."""
        e = sel.nonzero(as_tuple=True)[0]
        a = self.i[e]
        count = torch.bincount(a, minlength=self.n)
        rank = torch.arange(len(e), device=e.device) - (torch.cumsum(count, 0) - count)[a]
        tab = torch.zeros((self.n, 3), dtype=torch.long, device=e.device)
        q = rank < 3
        tab[a[q], rank[q]] = e[q]
        return tab, count.clamp(max=3)

    def embed(self, rho):
        p = self.p
        lo, hi = 0.85 * p.rhoe, 1.15 * p.rhoe
        s = p.rhoei * 1.176471
        x, y, z = rho * s - 1, rho * p.rhoei - 1, (rho * p.rhoei).clamp(min=1e-300)
        F = torch.where(rho < lo, p.Fn[0] + x * (p.Fn[1] + x * (p.Fn[2] + x * p.Fn[3])),
                        torch.where(rho < hi, p.F[0] + y * (p.F[1] + y * (p.F[2] + y * p.F[3])),
                                    p.Fe * (1 - p.eta * z.log()) * z ** p.eta))
        dF = torch.where(rho < lo, s * (p.Fn[1] + x * (2 * p.Fn[2] + 3 * x * p.Fn[3])),
                         torch.where(rho < hi, p.rhoei * (p.F[1] + y * (2 * p.F[2] + 3 * y * p.F[3])),
                                     -p.Fe * p.eta ** 2 * p.rhoei * z ** (p.eta - 1) * z.log()))
        return F, dF

    def forces(self, r):
        """Accelerations and per-atom energies over the list built last."""
        p, n, m, i, k = self.p, self.n, self.m, self.i, self.k
        F = torch.zeros((n, 3), dtype=torch.float64, device=r.device)
        U = torch.zeros(n, dtype=torch.float64, device=r.device)
        d = _wrap(r[i] - r[k], self.L)
        rr = (d * d).sum(1)
        if m:
            e = ((i < m) & (k < m) & (rr < p.rrCutEam)).nonzero(as_tuple=True)[0]
            a, b, R = i[e], k[e], rr[e].sqrt()
            x = R * p.rei
            eA, eB = torch.exp(-p.alpha * (x - 1)), torch.exp(-p.beta * (x - 1))
            uk, ul = x - p.kappa, x - p.lambda_
            dA, dB = 1 + uk ** 20, 1 + ul ** 20
            tA, tB = p.alpha + 20 * uk ** 19 / dA, p.beta + 20 * ul ** 19 / dB
            phi = p.A * eA / dA - p.B * eB / dB
            dphi = (-p.A * eA * tA / dA + p.B * eB * tB / dB) * p.rei
            f, df = p.fe * eB / dB, -p.fe * p.rei * eB * tB / dB
            rho = torch.zeros(n, dtype=torch.float64, device=r.device).index_add_(0, a, f)
            Fv, dF = self.embed(rho[:m])
            fc = -(dphi + df * (dF[a] + dF[b])) / R
            F.index_add_(0, a, fc[:, None] * d[e])
            U.index_add_(0, a, 0.5 * phi)
            U[:m] += Fv
        close_c = (i >= m) & (k >= m) & (rr < p.rrCutC)
        if m < n:
            # the first three close carbons of a carbon atom, and what is near a close carbon
            tab, cnt = self._three(close_c)
            tab2, cnt2 = self._three((i >= m) & (rr < p.rrCutC))
            p2 = torch.where(cnt == 3, self.j[tab[:, 2]], torch.full_like(cnt, -1))
        # Lennard-Jones; a carbon atom's list walk resumes at entry 4 after its third close carbon
        e = (((i < m) != (k < m)) & (rr < p.rrCutLJ)).nonzero(as_tuple=True)[0]
        if len(e):
            a, j = i[e], self.j[e]
            w = torch.ones(len(e), dtype=torch.float64, device=r.device)
            carbon = a >= m
            w[carbon & (j == 3) & (p2[a] == 2)] = 0
            w[carbon & (j >= 4) & (j <= p2[a])] = 2
            q = p.sigmaLJ ** 2 / rr[e]
            q3 = q ** 3
            F.index_add_(0, a, (w * 48 * p.epsLJ * q3 * (q3 - 0.5) / rr[e])[:, None] * d[e])
            U.index_add_(0, a, 0.5 * w * 4 * p.epsLJ * q3 * (q3 - 1))
        if m < n:
            for q in range(3):
                c = (cnt > q).nonzero(as_tuple=True)[0]          # atoms that have a close carbon q
                e = tab[c, q]
                rn, R = d[e], rr[e].sqrt()
                b = k[e]
                seen = torch.zeros_like(c)
                for t in range(3):                              # its first two others
                    e2 = tab2[b, t]
                    other = k[e2]
                    use = (cnt2[b] > t) & (other != c) & (seen < 2)
                    seen = seen + use
                    g = -d[e2]
                    den = R * rr[e2]
                    cs = torch.where(use, (rn * g).sum(1) / den, torch.zeros_like(R))
                    tmp = p.mu_theta * (torch.acos(cs) - p.theta_0) / (1 - cs * cs).sqrt()
                    f = (tmp / den)[:, None] * g - (tmp * cs / (R * R))[:, None] * rn
                    f[:, 2] -= p.mu_p * (r[other, 2] - p.z_0) / 9
                    F.index_add_(0, c[use], f[use])
            c = (cnt == 3).nonzero(as_tuple=True)[0]
            rn = [d[tab[c, q]] for q in range(3)]
            R = [rr[tab[c, q]].sqrt() for q in range(3)]
            f, u = torch.zeros_like(rn[0]), torch.zeros_like(R[0])
            for q in range(3):
                s = (q + 1) % 3
                cs = (rn[q] * rn[s]).sum(1) / (R[q] * R[s])
                dth = torch.acos(cs) - p.theta_0
                tmp = p.mu_theta * dth / (1 - cs * cs).sqrt() / (R[q] * R[s])
                f += (tmp * (1 - R[q] * cs / R[s]))[:, None] * rn[s] + (tmp * (1 - R[s] * cs / R[q]))[:, None] * rn[q]
                f -= (p.mu_r * (R[q] - 1) / R[q])[:, None] * rn[q]
                u += p.mu_theta * dth * dth + p.mu_r * (R[q] - 1) ** 2
            zs = sum(r[k[tab[c, q]], 2] - p.z_0 for q in range(3))
            z = r[c, 2] - p.z_0
            f[:, 2] -= 2.0 / 3.0 * p.mu_p * (2 * z - zs)
            u += p.mu_p * (z - zs / 3) ** 2
            F.index_add_(0, c, f)
            U.index_add_(0, c, 0.5 * u)
        F[:m] /= p.massMe
        return F, U


def _steps64(case, p, r, v):
    """The block of steps of one system in 64 bits: r with U, v, a, and the record's energies."""
    dev = _dev()
    r = torch.from_numpy(r[:, :3].astype(np.float64)).to(dev)
    v = torch.from_numpy(v.astype(np.float64)).to(dev)
    a, M = torch.zeros_like(v), _Model64(p, r)
    m, dt = p.nMolMe, p.deltaT
    c30 = float(np.float32(math.cos(math.pi / 6.0)))
    f32 = np.float32
    xl, xr = float(f32(0.5) * (f32(c30) - f32(p.region.x))), float(f32(0.5) * (f32(p.region.x) - f32(c30)))
    yb, yt = float(f32(0.5) * (f32(1) - f32(p.region.y))), float(f32(0.5) * (f32(p.region.y) - f32(1)))

    def moving():
        ok = (r[:, 0] != xl) & (r[:, 0] < xr) & (r[:, 1] != yt) & (r[:, 1] != yb)
        ok[:m] = True
        return ok.double()[:, None]

    rebuild, disp, scale = True, 0.0, None
    for sc in range(1, case["steps"] + 1):
        if scale is not None:
            v = v * scale
        f = moving()
        v = v + f * 0.5 * dt * a
        r = r + f * dt * v
        r = r - M.L * ((r >= 0.5 * M.L).double() - (r < -0.5 * M.L).double())
        if rebuild or case["rebuild"]:
            M.build(r)
            rebuild, disp = False, 0.0
        a, U = M.forces(r)
        v = v + moving() * 0.5 * dt * a
        vv = (v * v).sum(1)
        vm = v[:m].clone()
        if m and p.iRegime == 2:
            vm[:, 0] -= vm[:, 0].mean()
        vv_sum = vv[m:].sum() + p.massMe * (vm * vm).sum()
        kin = 0.5 * vv_sum / p.nMol
        disp += float(vv.max().sqrt()) * dt
        rebuild = rebuild or disp > 0.5 * p.rNebrShell
        scale = None
        if p.iRegime == 2 and sc > p.stepEquil and sc % p.stepThermostat == 0:
            scale = torch.ones((p.nMol, 1), dtype=torch.float64, device=dev)
            scale[m:] = torch.sqrt(1 + p.gammaBerendsen * (p.temperature * 1.5 * p.kB / kin - 1))
            if sc < p.stepEquil + p.stepCool:
                scale[:m] = torch.sqrt(1 + p.gammaBerendsen * (p.temperature * p.kB / kin - 1))
    if scale is not None:
        v = v * scale
    pe = U.sum() / p.nMol
    rec = torch.stack([kin, pe, kin + pe, vv_sum, vv.max(), U.sum()])
    return torch.cat([r, U[:, None]], 1), v, a, rec


def _splines64(q, theta, R):
    """phi and f of theta at R: uniform cubic B-splines on 29 intervals from 0.6 r_e to the cutoff."""
    r0, h = 0.6 / q.rei, (math.sqrt(q.rrCutEam) - 0.6 / q.rei) / 29
    x = (R - r0) / h
    k = x.detach().floor().clamp(0, 28).long()
    t = x - k
    b = [(1 - t) ** 3 / 6, (3 * t ** 3 - 6 * t ** 2 + 4) / 6, (-3 * t ** 3 + 3 * t ** 2 + 3 * t + 1) / 6, t ** 3 / 6]
    return (sum(theta[2 + k + s] * b[s] for s in range(4)), sum(theta[34 + k + s] * b[s] for s in range(4)))


def _frame64(q, r, theta, ref, what, natoms):
    """One frame: its energy, forces, loss and gradient, as the case asks."""
    dev = _dev()
    x = torch.from_numpy(r[:, :3].astype(np.float64)).to(dev)
    M = _Model64.__new__(_Model64)
    M.p, M.n, M.m = q, q.nMol, q.nMolMe
    M.L = torch.tensor([q.region.x, q.region.y, q.region.z], dtype=torch.float64, device=dev)
    metal, L = M.m, M.L
    # pairs (metal, any) within the larger cutoff
    cut = math.sqrt(max(q.rrCutEam, q.rrCutLJ))
    I, K = [], []
    for b in range(0, metal, 512):
        d = _wrap(x[b:min(b + 512, metal), None].float().double() - x[None], L)
        i, k = ((d * d).sum(2) < cut * cut).nonzero(as_tuple=True)
        i = i + b
        keep = (i != k) & ((k >= metal) | (i < k))
        I.append(i[keep])
        K.append(k[keep])
    I, K = torch.cat(I), torch.cat(K)
    with torch.enable_grad():
        x = x.requires_grad_(what != "energy_grad")
        d = _wrap((x[I] - x[K]).detach(), L) + ((x[I] - x[K]) - (x[I] - x[K]).detach())
        rr = (d * d).sum(1)
        e = ((K < metal) & (rr < q.rrCutEam)).nonzero(as_tuple=True)[0]
        phi, f = _splines64(q, theta, rr[e].sqrt())
        rho = torch.zeros(metal, dtype=torch.float64, device=dev).index_add(0, I[e], f).index_add(0, K[e], f)
        E = phi.sum() + M.embed(rho)[0].sum()
        e = ((K >= metal) & (rr < q.rrCutLJ)).nonzero(as_tuple=True)[0]
        s6 = (theta[1] ** 2 / rr[e]) ** 3
        E = E + (4 * theta[0] * (s6 * s6 - s6)).sum()
        if what == "energy_grad":
            return E.detach(), torch.autograd.grad(E, theta)[0]
        g, = torch.autograd.grad(E, x, create_graph=what == "loss_grad")
        if what == "forces":
            return -g.detach(), None
        loss = ((-g - torch.from_numpy(ref.astype(np.float64)).to(dev)) ** 2).sum() / (3 * natoms)
        return loss.detach(), torch.autograd.grad(loss, theta)[0]


def exact(case, seed):
    kind = case["kind"]
    if kind == "rdf":
        return None
    if kind == "diff":
        q, frames = _frames(case, seed)
        theta, ref = _theta_ref(case, seed, q, q.nMol * case["frames"])
        th = torch.tensor(theta, dtype=torch.float64, device=_dev(), requires_grad=True)
        got = [_frame64(q, r, th, ref[k * q.nMol:(k + 1) * q.nMol], case["what"], q.nMol * len(frames))
               for k, r in enumerate(frames)]
        if case["what"] == "forces":
            return {"forces": torch.cat([g[0] for g in got])}
        grad = sum(g[1] for g in got)
        if case["what"] == "energy_grad":
            return {"energy": torch.stack([g[0] for g in got]), "grad": grad}
        return {"loss": sum(g[0] for g in got).reshape(1), "grad": grad}
    systems = [_system(case, seed)] if kind == "noalloc" else _systems(case, seed)
    if max(s[0].nMol for s in systems) > _MOST_ATOMS:
        return None
    if kind == "noalloc":
        p, r, _ = systems[0]
        x = torch.from_numpy(r[:, :3].astype(np.float64)).to(_dev())
        M = _Model64(p, x)
        M.build(x)
        a, U = M.forces(x)
        return {"pos": torch.cat([x, U[:, None]], 1), "acc": torch.cat([a, torch.zeros_like(U)[:, None]], 1)}
    got = [_steps64(case, *s) for s in systems]
    return {"r": torch.cat([g[0] for g in got]), "v": torch.cat([g[1] for g in got]),
            "a": torch.cat([g[2] for g in got]), "thermo": got[0][3]}
