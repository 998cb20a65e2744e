"""The work that a fitting run has this framework do, as cases that can be timed and checked.

A case is a training set (kind, configurations, sizes), a population and the entry point that is
called on them:

  fitness   Fitness.compute: one generation's fitness of a host population, into the caller's FP32
            buffer as the reference's GA holds it (Fitness::compute(int, float*, float*))
  forces    Fitness.batched_forces: the per-atom forces of a handful of candidates
  ga        GA.advance + GA.state: whole generations (fitness, selection, crossover, mutation)
  predict   Fitness.find_force64: FP64 forces, virials and energies of one parameter vector

prepare() makes what a program holds before the call: the engine with its training set and the
population.  exact() evaluates the same inputs in plain FP64 torch.
"""
import math

import numpy as np
import torch

from gpuga_b200 import GA, Fitness

DEV = "cuda"
F64 = torch.float64

# ------------------------------------------------------------------------------------ structures
DIAMOND = [[0, 0, 0], [0, .5, .5], [.5, 0, .5], [.5, .5, 0], [.25, .25, .25], [.25, .75, .75], [.75, .25, .75],
           [.75, .75, .25]]
FCC = [[0, 0, 0], [0, .5, .5], [.5, 0, .5], [.5, .5, 0]]
FLUORITE = FCC + [[x, y, z] for x in (.25, .75) for y in (.25, .75) for z in (.25, .75)]
WURTZITE = [[1 / 3, 2 / 3, 0], [2 / 3, 1 / 3, .5], [1 / 3, 2 / 3, .382], [2 / 3, 1 / 3, .882]]
# wurtzite and fluorite supercells of 96 to 324 atoms (thinner than twice the 8 A cutoff in places)
WURTZITE_REPS = [(4, 3, 2), (3, 3, 3), (4, 4, 2), (3, 3, 4), (4, 4, 3), (5, 5, 2), (3, 3, 6), (5, 4, 3), (4, 4, 4),
                 (6, 4, 3), (9, 3, 3)]
FLUORITE_REPS = [(2, 2, 2), (3, 2, 2), (4, 2, 2), (3, 3, 2), (4, 3, 2), (3, 3, 3)]

# potential.in bounds: the Si example of the reference, its two-element GaAs example and the
# rigid-ion oxide bounds of the benchmark set; networks search every weight in [-3, 3]
SI = [[2.9, 3.3], [1.3, 1.5], [2.2, 2.4], [2, 2], [0.5, 0.8], [0, 0.4], [-0.8, -0.6], [2.8, 2.8], [3.2, 3.2]]
GAAS = [[2.7, 3.3], [1.0, 1.5], [2.2, 2.4], [1.5, 2.5], [2.8, 3.3], [1.0, 1.5], [2.2, 2.4], [1.5, 2.5], [0.5, 1.5],
        [0.1, 0.5], [-1, -0.5], [2.9, 2.9], [3.2, 3.2]]
OXIDE = [[2.0, 2.6], [0, 0], [1, 1], [0, 0], [1000, 3000], [0.25, 0.35], [0, 50], [10000, 25000], [0.12, 0.20],
         [10, 40], [8, 8], [0, 0.5], [1, 2], [2.0, 2.5], [2, 2]]


def supercell(frac, cell, reps):
    shift = np.array([[i, j, k] for i in range(reps[0]) for j in range(reps[1]) for k in range(reps[2])], np.float64)
    n = np.array(reps, np.float64)
    return ((np.array(frac)[None] + shift[:, None]) / n).reshape(-1, 3), np.array(cell, np.float64) * n[:, None]


def one_structure(case, rng):
    """(fractional positions, cell, types, largest isotropic strain, displacement sigma) of one configuration;
    rng chooses its size, alike for every seed of a case."""
    kind = case["kind"]
    if kind == "si":
        n = int(rng.integers(case["min_rep"], case["max_rep"] + 1))
        frac, cell = supercell(DIAMOND, np.eye(3) * 5.43, (n, n, n))
        return frac, cell, np.zeros(len(frac)), 0.03, case["sigma"]
    if kind == "polytypes":  # up to 4, 6, 12 and 14 neighbors
        unit, a = [(DIAMOND, 5.43), ([[0, 0, 0]], 2.53), (FCC, 3.9), ([[0, 0, 0], [.5, .5, .5]], 3.08)][rng.integers(4)]
        n = int(rng.integers(2, 4)) + (2 if len(unit) < 4 else 0)
        frac, cell = supercell(unit, np.eye(3) * a, (n, n, n))
        return frac, cell, np.zeros(len(frac)), 0.02, case["sigma"]
    if kind == "gaas":
        n = int(rng.integers(case["min_rep"], case["max_rep"] + 1))
        frac, cell = supercell(DIAMOND, np.eye(3) * 5.65, (n, n, n))
        return frac, cell, np.tile([0, 0, 0, 0, 1, 1, 1, 1], n ** 3), 0.03, case["sigma"]
    if kind == "oxide":
        if rng.uniform() < 0.5:
            reps = WURTZITE_REPS[rng.integers(len(WURTZITE_REPS))]
            cell = [[3.25, 0, 0], [-3.25 / 2, 3.25 * math.sqrt(3) / 2, 0], [0, 0, 5.21]]
            frac, cell = supercell(WURTZITE, cell, reps)
            return frac, cell, np.tile([0, 0, 1, 1], int(np.prod(reps))), 0.02, case["sigma"]
        reps = FLUORITE_REPS[rng.integers(len(FLUORITE_REPS))]
        frac, cell = supercell(FLUORITE, np.eye(3) * 5.10, reps)
        return frac, cell, np.tile([0] * 4 + [1] * 8, int(np.prod(reps))), 0.02, case["sigma"]
    if case.get("dimers") and rng.uniform() < 0.5:  # two atoms in a wide box
        d = rng.uniform(2.0, 7.5) / 20.0
        return np.array([[.4, .4, .4], [.4 + d, .4, .4]]), np.eye(3) * 20.0, np.zeros(2), 0.0, 0.0
    n = int(rng.integers(2, 4))
    frac, cell = supercell(DIAMOND, np.eye(3) * 5.43, (n, n, n))
    return frac, cell, np.zeros(len(frac)), 0.0, case["sigma"]


def spec_of(case):
    kind = case["kind"]
    if kind in ("si", "polytypes"):
        s = dict(potential_type=1, cutoff=3.0 if kind == "si" else 3.2, weights=(0.05, 0.15, 0.8), bounds=SI)
    elif kind == "gaas":
        s = dict(potential_type=2, cutoff=3.2, weights=(0.3, 0.3, 0.4), bounds=GAAS)
    elif kind == "oxide":
        s = dict(potential_type=4 if case["neutral"] else 0, cutoff=8.0, weights=(0.1, 0.2, 0.7), bounds=OXIDE)
    else:
        n = case["neurons"]
        s = dict(potential_type=3, cutoff=case["taper_end"], weights=(0.4, 0.3, 0.3),
                 bounds=[[-3.0, 3.0]] * (n * (n + 4) + 1))
    s["bounds"] = np.array(s["bounds"], np.float32)
    return s


def decode(spec, x01):
    """FP32 parameters of x in [0, 1], as the reference decodes them, in FP64."""
    lo, hi = spec["bounds"][:, 0], spec["bounds"][:, 1]
    return (lo + ((hi - lo) * x01.astype(np.float32)).astype(np.float32)).astype(np.float32).astype(np.float64)


# ------------------------------------------------------------------- training sets and their lists
class Group:
    """The configurations of one size: padded neighbor lists and bond vectors, in FP64 on the GPU."""

    def __init__(self, cfgs, starts, na, pos, box, types, cutoff):
        self.cfgs, self.na, self.m = cfgs, na, len(cfgs)
        self.atoms = np.concatenate([np.arange(starts[c], starts[c] + na) for c in cfgs])
        r = torch.from_numpy(pos[self.atoms]).to(DEV, F64).view(self.m, na, 3)
        cell = torch.from_numpy(box[cfgs]).to(DEV, F64)  # rows: cell vectors
        inv = torch.linalg.inv(cell)
        self.type = torch.from_numpy(types[self.atoms]).to(DEV).view(self.m, na)
        near, step = [], max(1, 4_000_000 // (na * na))
        for a in range(0, self.m, step):
            x = r[a:a + step]
            v = x[:, None, :, :] - x[:, :, None, :]  # [m, i, j]: r_j - r_i
            s = v @ inv[a:a + step, None]
            v = (s - torch.round(s)) @ cell[a:a + step, None]
            near.append((v.square().sum(-1) < cutoff * cutoff) & ~torch.eye(na, dtype=torch.bool, device=DEV))
        near = torch.cat(near)
        self.z = max(1, int(near.sum(-1).max()))
        self.idx = torch.argsort((~near).to(torch.uint8), dim=-1, stable=True)[..., :self.z]
        self.mask = torch.gather(near, -1, self.idx)
        at = torch.arange(self.m, device=DEV)[:, None, None]
        v = r[at, self.idx] - r[:, :, None, :]
        s = torch.einsum("mizc,mcd->mizd", v, inv)
        self.v = torch.einsum("mizc,mcd->mizd", s - torch.round(s), cell)
        self.v = torch.where(self.mask[..., None], self.v, torch.ones((), dtype=F64, device=DEV))
        self.d = self.v.square().sum(-1).sqrt()
        self.u = self.v / self.d[..., None]

    def reverse(self):
        """Flat position (config, atom, slot) of every bond's reverse."""
        at = torch.arange(self.m, device=DEV)[:, None, None]
        back = self.idx[at, self.idx] == torch.arange(self.na, device=DEV)[None, :, None, None]  # [m, i, z, z']
        back &= self.mask[at, self.idx]
        return (at * self.na + self.idx) * self.z + back.to(torch.uint8).argmax(-1)


def taper(d, r1, r2):
    x = math.pi / (r2 - r1) * (d - r1)
    inside, shell = d < r1, (d >= r1) & (d < r2)
    one, zero = torch.ones_like(d), torch.zeros_like(d)
    return (torch.where(inside, one, torch.where(shell, 0.5 * torch.cos(x) + 0.5, zero)),
            torch.where(shell, -0.5 * math.pi / (r2 - r1) * torch.sin(x), zero))


def evaluate_tersoff(g, par, two, want):
    off = 4 if two else 0
    col = lambda k: par[:, k].view(-1, 1, 1, 1)  # noqa: E731
    n, beta, h = col(4 + off), col(5 + off), col(6 + off)
    fc, fcp = taper(g.d, float(par[0, 7 + off]), float(par[0, 8 + off]))  # R1, R2 are fixed by the bounds
    fc, fcp = fc * g.mask, fcp * g.mask
    other = g.mask[..., None] & g.mask[..., None, :] & ~torch.eye(g.z, dtype=torch.bool, device=DEV)
    cos = torch.einsum("mizc,miyc->mizy", g.u, g.u) * other
    w = fc[:, :, None, :] * other
    s2, s1, s0 = (w * cos * cos).sum(-1), (w * cos).sum(-1), w.sum(-1)
    zeta = beta * (s2 - 2 * h * s1 + h * h * s0)
    low = zeta < 1e-16
    zs = torch.where(low, torch.ones_like(zeta), zeta)
    zn = zs ** n
    b = torch.where(low, torch.ones_like(zeta), (1 + zn) ** (-0.5 / n))
    db = torch.where(low, torch.zeros_like(zeta), -0.5 * b * zn / ((1 + zn) * zs))
    del zn, zs
    unlike = (g.type[:, :, None] != g.type[torch.arange(g.m, device=DEV)[:, None, None], g.idx]) if two else None
    pick = lambda k: torch.where(unlike, col(4 + k), col(k)) if two else col(k)  # noqa: E731
    D0, al, r0, S = pick(0), pick(1), pick(2), pick(3)
    lr, la, t = torch.sqrt(2 * S) * al, torch.sqrt(2 / S) * al, g.d - r0
    fr, fa = D0 / (S - 1) * torch.exp(-lr * t), S * D0 / (S - 1) * torch.exp(-la * t)
    e = fr - b * fa
    site = 0.5 * (fc * e).sum(-1)
    dA = fcp * e + fc * (-lr * fr + b * la * fa)
    Sj = db * fa
    del fr, fa, b, db, zeta
    T = Sj * fc
    c2, u3 = cos * cos, g.u[:, :, None, :, :] * other[..., None]
    Tc2, Tc, T0 = (torch.einsum("pmik,mijk->pmij", T, x) for x in (c2, cos, other.to(F64)))
    sum_g = beta * (Tc2 - 2 * h * Tc + h * h * T0)
    sum_q = beta * (Sj * (s2 - h * s1) + Tc2 - h * Tc)
    X1, X0 = ((w * cos)[..., None] * u3).sum(-2), (w[..., None] * u3).sum(-2)
    V = Sj[..., None] * (X1 - h[..., None] * X0) + torch.einsum("pmik,mijkc->pmijc", T, cos[..., None] * u3)
    V = beta[..., None] * (V - h[..., None] * torch.einsum("pmik,mijkc->pmijc", T, u3))
    m = -2 * fc / g.d
    f = 0.5 * ((dA - fcp * sum_g - m * sum_q)[..., None] * g.u + m[..., None] * V) * g.mask[..., None]
    out = {"pe": site}
    if "W" in want:  # configuration virial -sum r_ij (x) f_ij
        out["W"] = torch.stack([-(g.v[..., a] * f[..., c]).sum((-1, -2)) for a, c in
                                ((0, 0), (1, 1), (2, 2), (0, 1), (1, 2), (2, 0))], -1)
    if "F" in want or "Wi" in want:
        flat = f.reshape(f.shape[0], -1, 3)
        df = (flat - flat[:, g.reverse().reshape(-1)]).view_as(f) * g.mask[..., None]
        out["F"] = df.sum(-2)
        if "Wi" in want:
            out["Wi"] = torch.stack([-0.5 * (g.v[..., a] * df[..., c]).sum(-1) for a, c in
                                     ((0, 0), (1, 1), (2, 2), (0, 1), (1, 2), (2, 0))], -1)
    return out


def pair_sums(g, U, dU, want):
    U, dU = U * g.mask, dU * g.mask
    out = {"pe": 0.5 * U.sum(-1)}
    if "F" in want:
        out["F"] = torch.einsum("pmiz,mizc->pmic", dU, g.u)
    if "W" in want:
        s = -0.5 * dU * g.d
        out["W"] = torch.stack([(s * (g.u[..., a] * g.u[..., c])).sum((-1, -2)) for a, c in
                                ((0, 0), (1, 1), (2, 2), (0, 1), (1, 2), (2, 0))], -1)
    return out


def evaluate_oxide(g, par, neutral, self_energy, want):
    ratio, kc, alpha = (-1.0 if neutral else -0.5), 14.399645, 0.2
    two_pi = 2 * alpha / math.sqrt(math.pi)
    t = g.type[:, :, None] + g.type[torch.arange(g.m, device=DEV)[:, None, None], g.idx]
    q2 = kc * par[:, :1].square()
    table = lambda x: x[:, t.reshape(-1)].view(x.shape[0], *t.shape)  # noqa: E731  [p, 3] -> per pair
    A, irho, C = (table(x) for x in (par[:, [1, 4, 7]], 1 / par[:, [2, 5, 8]], par[:, [3, 6, 9]]))
    qq = table(torch.cat([q2, ratio * q2, ratio * ratio * q2], 1))
    rc = float(par[0, 10])  # fixed by the bounds
    v = math.erfc(alpha * rc) / rc
    dv = -v / rc - two_pi * math.exp(-(alpha * rc) ** 2) / rc
    ec = torch.erfc(alpha * g.d) / g.d
    gc = ec / g.d + two_pi * torch.exp(-(alpha * g.d).square()) / g.d
    i6 = g.d ** -6
    buck = A * torch.exp(-g.d * irho)
    U = buck - C * i6 + qq * (ec - v - dv * (g.d - rc))
    dU = -irho * buck + 6 * C * (i6 / g.d) - qq * (gc + dv)
    del buck, A, irho, C, qq
    D0, al, r0, S = (par[:, k].view(-1, 1, 1, 1) for k in (11, 12, 13, 14))
    lr, la, x = torch.sqrt(2 * S) * al, torch.sqrt(2 / S) * al, g.d - r0
    fr, fa = D0 / (S - 1) * torch.exp(-lr * x), S * D0 / (S - 1) * torch.exp(-la * x)
    U, dU = U + (fr - fa) * (t == 1), dU + (la * fa - lr * fr) * (t == 1)
    out = pair_sums(g, U, dU, want)
    if self_energy:
        k = alpha / math.sqrt(math.pi) + v + 0.5 * two_pi * math.exp(-(alpha * rc) ** 2)
        charge = torch.where(g.type == 0, 1.0, ratio * ratio).to(F64)
        out["pe"] = out["pe"] - q2.view(-1, 1, 1) * k * charge
    return out


def evaluate_network(g, par, n, r1, r2, want):
    fc, fcp = taper(g.d, r1, r2)
    U, dU = [], []
    for w in par:
        w0, b0, W1, b1, w2, b2 = torch.split(w, [n, n, n * n, n, n, 1])
        x1 = torch.tanh(g.d[..., None] * w0 - b0)
        y1 = (1 - x1 * x1) * w0
        W1 = W1.view(n, n).T
        x2 = torch.tanh(x1 @ W1 - b1)
        u = (x2 @ w2 - b2) * fc  # the reference tapers the energy before it enters the force
        U.append(u)
        dU.append((((1 - x2 * x2) * (y1 @ W1)) @ w2) * fc + u * fcp)
    return pair_sums(g, torch.stack(U), torch.stack(dU), want)


def evaluate(case, g, par, want):
    """Per chunk of parameter vectors: pe [p, m, na], F [p, m, na, 3], W [p, m, 6] of the group, in FP64."""
    kind = case["kind"]
    per = g.m * g.na * g.z * {"si": 40, "polytypes": 60, "gaas": 60, "oxide": 20}.get(kind, 4 * case.get("neurons", 1))
    step = max(1, 400_000_000 // per)
    for a in range(0, len(par), step):
        x = par[a:a + step]
        if kind == "oxide":
            yield a, evaluate_oxide(g, x, case["neutral"], case["self_energy"], want)
        elif kind == "network":
            yield a, evaluate_network(g, x, case["neurons"], case["taper_start"], case["taper_end"], want)
        else:
            yield a, evaluate_tersoff(g, x, kind == "gaas", want)


class TrainingSet:
    """Seeded configurations with their targets from a teacher parameter vector, in the layouts of
    Fitness(arrays=...)."""

    def __init__(self, case, seed):
        rng, sizes = np.random.default_rng(seed), np.random.default_rng([case["configs"], case["population"]])
        self.spec = spec = spec_of(case)
        pos, box, types, na = [], [], [], []
        for _ in range(case["configs"]):
            frac, cell, t, strain, sigma = one_structure(case, sizes)
            cell = cell * (1 + rng.uniform(-strain, strain))
            pos.append(frac @ cell + rng.normal(0, 1, (len(frac), 3)) * sigma)
            box.append(cell)
            types.append(t)
            na.append(len(frac))
        self.na = np.array(na, np.int32)
        self.nc, self.ncf, self.n = len(na), case["force_configs"], int(self.na.sum())
        self.nf = int(self.na[:self.ncf].sum())
        pos, box = np.concatenate(pos).astype(np.float32), np.array(box, np.float32)
        types = np.concatenate(types).astype(np.int64)
        self.starts = np.concatenate([[0], np.cumsum(self.na)[:-1]])
        d = len(spec["bounds"])
        if case["kind"] == "network":  # weights N(0, 0.3)
            self.teacher = np.clip((rng.normal(0, 0.3, d) + 3) / 6, 0, 1).astype(np.float32)
        else:
            self.teacher = rng.uniform(0, 1, d).astype(np.float32)
        p = case["population"]
        self.pop = rng.uniform(0, 1, (p, d)).astype(np.float32)
        if case["late"]:  # a converging population: scattered around the best parameters
            self.pop = np.clip(self.teacher + rng.normal(0, 0.05, (p, d)), 0, 1).astype(np.float32)
        self.groups = []
        for k in np.unique(self.na):
            for part in (np.arange(self.ncf), np.arange(self.ncf, self.nc)):
                cfgs = part[self.na[part] == k]
                if len(cfgs):
                    self.groups.append(Group(cfgs, self.starts, int(k), pos, box, types, spec["cutoff"]))
        par = torch.from_numpy(decode(spec, self.teacher[None])).to(DEV)
        self.pe_ref, self.w_ref = np.zeros(self.nc, np.float32), np.zeros((self.nc, 6), np.float32)
        self.f_ref = np.zeros((self.n, 3), np.float32)
        for g in self.groups:
            forces = g.cfgs[0] < self.ncf
            for _, r in evaluate(case, g, par, "F" if forces else "W"):
                if forces:
                    self.f_ref[g.atoms] = r["F"][0].reshape(-1, 3).cpu().numpy()
                else:
                    self.pe_ref[g.cfgs] = r["pe"][0].sum(-1).cpu().numpy()
                    self.w_ref[g.cfgs] = r["W"][0].cpu().numpy()
        self.arrays = dict(
            potential_type=spec["potential_type"], num_neurons=case.get("neurons", 0), cutoff=spec["cutoff"],
            w_force=spec["weights"][0], w_energy=spec["weights"][1], w_stress=spec["weights"][2],
            pmin=spec["bounds"][:, 0].copy(), pmax=spec["bounds"][:, 1].copy(), Na=self.na, Nc_force=self.ncf,
            type=types.astype(np.int32), r=np.ascontiguousarray(pos.T).reshape(-1), box9=box.reshape(-1),
            pe_ref=self.pe_ref, virial_ref=np.ascontiguousarray(self.w_ref.T).reshape(-1),
            force_ref=np.ascontiguousarray(self.f_ref.T).reshape(-1))


def engine_options(case):
    o = {}
    if case["kind"] == "network":
        o.update(nn2b_r1=case["taper_start"], nn2b_r2=case["taper_end"])
    if case["kind"] == "oxide":
        o.update(ri_self_energy=case["self_energy"])
    return o


# ----------------------------------------------------------------------------------------- the cases
def tersoff(name, entry, kind, configs, force_configs, population, min_rep=1, max_rep=4, sigma=0.1, late=False,
            generations=0):
    c = dict(entry=entry, kind=kind, configs=configs, force_configs=force_configs, population=population,
             min_rep=min_rep, max_rep=max_rep, sigma=sigma, late=late, generations=generations)
    return dict(c, name=name) if name else c


def oxide(name, entry, configs, population, neutral=False, self_energy=False, late=False):
    c = dict(entry=entry, kind="oxide", configs=configs, force_configs=configs // 2, population=population,
             sigma=0.08, neutral=neutral, self_energy=self_energy, late=late)
    return dict(c, name=name) if name else c


def network(name, entry, configs, population, neurons, taper_start, taper_end, dimers=False, late=False):
    c = dict(entry=entry, kind="network", configs=configs, force_configs=configs // 2, population=population,
             neurons=neurons, taper_start=taper_start, taper_end=taper_end, dimers=dimers, sigma=0.15, late=late)
    return dict(c, name=name) if name else c


def listed():
    return [
        # a first look at a potential: a handful of 8-atom cells, a small population; latency and launches
        tersoff("si_tiny", "fitness", "si", 6, 3, 20, max_rep=1),
        # the small GA run: 20 cells of 64 atoms, population 100, whole generations on the device loop
        tersoff("si_ga", "ga", "si", 20, 10, 100, min_rep=2, max_rep=2, sigma=0.05, generations=4),
        # the main fit: 500 configurations of 8 to 512 atoms (~1e5 atoms), population 1000
        tersoff("si_main", "fitness", "si", 500, 250, 1000),
        # late generations of a fit with few force configurations and cells of up to 1000 atoms, an odd population
        tersoff("si_late", "fitness", "si", 67, 5, 333, max_rep=5, late=True),
        # a set that mixes polytypes: 4, 6, 12 and 14 neighbors per atom
        tersoff("si_polytypes", "fitness", "polytypes", 60, 31, 150, sigma=0.06),
        # two elements, S a fitted parameter (the GaAs example's potential.in)
        tersoff("gaas", "fitness", "gaas", 100, 50, 200, min_rep=2, max_rep=3, sigma=0.08),
        # rigid ions: 300 oxide configurations of 96 to 324 atoms at an 8 A cutoff, population 400
        oxide("oxide_main", "fitness", 300, 400),
        # a small neutral oxide set with the self energy, near the optimum
        oxide("oxide_small", "fitness", 13, 50, neutral=True, self_energy=True, late=True),
        # network potential 1-16-16-1, 200 cells of 64 or 216 atoms, population 200
        network("network_16", "fitness", 200, 200, 16, 4.0, 5.0),
        # the reference's largest width and its 7-8 A taper, dimers among the cells
        network("network_10", "fitness", 31, 100, 10, 7.0, 8.0, dimers=True),
        # the forces of a few candidates, to be looked at one by one
        tersoff("si_forces", "forces", "si", 40, 20, 8, min_rep=2, max_rep=4, late=True),
        # the end of a run: the elite's forces, energies and virials in FP64 over the whole set
        tersoff("si_predict", "predict", "si", 500, 250, 1, late=True),
    ]


def draw(rng):
    spread = lambda lo, hi: int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))  # noqa: E731
    pick, late = rng.random(), rng.random() < 0.4
    if pick < 0.40:
        configs, max_rep = spread(4, 400), rng.randint(1, 5)
        most = 1e8 / (configs * sum(8 * n ** 3 for n in range(1, max_rep + 1)) / max_rep)
        return tersoff(None, "fitness", "si", configs, rng.randint(1, configs - 2),
                       min(spread(8, 1000), max(8, int(most))), max_rep=max_rep, sigma=rng.choice((0.05, 0.1)), late=late)
    if pick < 0.48:
        return tersoff(None, "fitness", "polytypes", spread(6, 80), 3, spread(8, 200), sigma=0.06, late=late)
    if pick < 0.58:
        configs = spread(4, 120)
        return tersoff(None, "fitness", "gaas", configs, rng.randint(1, configs - 2), spread(8, 300), min_rep=1,
                       max_rep=3, sigma=0.08, late=late)
    if pick < 0.74:
        return oxide(None, "fitness", spread(4, 250), spread(8, 400), rng.random() < 0.4, rng.random() < 0.4, late)
    if pick < 0.90:
        wide = rng.random() < 0.4
        r1, r2 = (7.0, 8.0) if wide else (4.0, 5.0)
        return network(None, "fitness", spread(4, 30 if wide else 160), spread(8, 200), rng.randint(4, 16), r1, r2,
                       wide and rng.random() < 0.5, late)
    if pick < 0.95:
        return tersoff(None, "forces", "si", spread(4, 60), 2, spread(1, 12), max_rep=rng.randint(2, 4), late=late)
    return tersoff(None, "predict", "si", spread(4, 500), 2, 1, max_rep=rng.randint(2, 4), late=True)


class State:
    pass


def prepare(case, seed):
    s = State()
    s.case = case
    ts = TrainingSet(case, seed)
    s.engine = Fitness(arrays=ts.arrays, **engine_options(case))
    s.p, s.pop = case["population"], np.ascontiguousarray(ts.pop)
    s.fitness = np.zeros(s.p, np.float32)
    if case["entry"] == "ga":
        s.ga = GA(s.engine, seed=seed % (1 << 31), population_size=s.p, parent_number=s.p // 2, mutation_rate=0.2,
                  maximum_generation=10_000_000)
    s.params = decode(ts.spec, s.pop[0])
    return s


def run(state):
    entry = state.case["entry"]
    if entry == "fitness":
        state.engine.compute(state.p, state.pop, state.fitness)
        return state.fitness
    if entry == "forces":
        return state.engine.batched_forces(state.pop)
    if entry == "ga":
        state.ga.advance(state.case["generations"])
        _, population, fitness = state.ga.state(state.p)
        return population, fitness
    return state.engine.find_force64(state.params)


def exact(case, seed):
    if case["entry"] == "ga":  # decided by random choices from the host's generator: no closed value
        return None
    ts = TrainingSet(case, seed)
    spec = ts.spec
    if case["entry"] == "predict":
        par = torch.from_numpy(decode(spec, ts.pop[:1])).to(DEV)
        F, W, pe = np.zeros((ts.n, 3)), np.zeros((ts.n, 6)), np.zeros(ts.n)
        for g in ts.groups:
            for _, r in evaluate(case, g, par, ("F", "Wi")):
                F[g.atoms] = r["F"][0].reshape(-1, 3).cpu().numpy()
                W[g.atoms] = r["Wi"][0].reshape(-1, 6).cpu().numpy()
                pe[g.atoms] = r["pe"][0].reshape(-1).cpu().numpy()
        return np.ascontiguousarray(F.T).reshape(-1), np.ascontiguousarray(W.T).reshape(-1), pe
    par = torch.from_numpy(decode(spec, ts.pop)).to(DEV)
    if case["entry"] == "forces":
        F = np.zeros((ts.pop.shape[0], 3, ts.nf))
        for g in ts.groups:
            if g.cfgs[0] < ts.ncf:
                for a, r in evaluate(case, g, par, "F"):
                    x = r["F"]
                    F[a:a + len(x), :, g.atoms] = x.reshape(len(x), -1, 3).cpu().numpy().transpose(0, 2, 1)
        return F
    e2, w2, f2 = (torch.zeros(len(par), dtype=F64, device=DEV) for _ in range(3))
    for g in ts.groups:
        forces = g.cfgs[0] < ts.ncf
        f_ref = torch.from_numpy(ts.f_ref[g.atoms]).to(DEV, F64).view(g.m, g.na, 3)
        pe_ref, w_ref = (torch.from_numpy(x[g.cfgs]).to(DEV, F64) for x in (ts.pe_ref, ts.w_ref))
        for a, r in evaluate(case, g, par, "F" if forces else "W"):
            p = slice(a, a + r["pe"].shape[0])
            if forces:
                f2[p] += (r["F"] - f_ref).square().sum((-1, -2, -3))
            else:
                e2[p] += (r["pe"].sum(-1) - pe_ref).square().sum(-1)
                w2[p] += (r["W"] - w_ref).square().sum((-1, -2))
    pe, w = ts.pe_ref[ts.ncf:].astype(np.float64), ts.w_ref[ts.ncf:].astype(np.float64)
    lowest = min(0.0, float(pe.min())) if len(pe) else 0.0
    wf, we, ws = (float(np.float32(x)) for x in spec["weights"])
    fit = we * torch.sqrt(e2 / float(np.square(pe - lowest).sum())) + ws * torch.sqrt(w2 / float(np.square(w).sum()))
    fit = fit + wf * torch.sqrt(f2 / float(np.square(ts.f_ref[:ts.nf].astype(np.float64)).sum()))
    return fit.cpu().numpy()


def atoms_of(case):
    """Mean (atoms, neighbors per atom) of a case's configurations."""
    kind = case["kind"]
    if kind in ("si", "gaas"):
        reps = range(case["min_rep"], case["max_rep"] + 1)
        return sum(8 * n ** 3 for n in reps) / len(reps), 4
    if kind == "polytypes":
        return 110, 9
    if kind == "oxide":
        return 185, 146
    shell = 4 / 3 * math.pi * case["taper_end"] ** 3 * 8 / 5.43 ** 3
    return (70, shell) if case["dimers"] else (140, shell)


def work(case):
    na, z = atoms_of(case)
    n, p, d = case["configs"] * na, case["population"], len(spec_of(case)["bounds"])
    if case["kind"] == "oxide":  # per unordered pair: one exponential, the three-term force, its share of the rest
        flops = z / 2 * 40
    elif case["kind"] == "network":  # per unordered pair: the two layers forward with their derivative
        k = case["neurons"]
        flops = z / 2 * (4 * k * k + 13 * k + 10 + 2 * k * 8)
    else:  # per bond: pair terms and bond order; per ordered triplet: cosine and three-body force
        flops = 60 * z + 4 * 8 * z + 21 * z * (z - 1)
    forces = case["configs"] and n * case["force_configs"] / case["configs"]
    read = 16 * n + 12 * forces + 64 * case["configs"] + 4 * p * d
    runs = max(1, case.get("generations", 0))
    if case["entry"] == "forces":
        return {"bytes": 16 * forces + 12 * p * forces, "flops": flops * forces * p}
    if case["entry"] == "predict":
        return {"bytes": read + 80 * n, "flops": flops * n}
    return {"bytes": runs * (read + 4 * p), "flops": runs * flops * n * p}
