"""The work this engine is measured on: Monte Carlo energies of one system, and batches of chains.

A case names an operation, a seeded synthetic system (the generators of mc_cpp_gb300.systems, with
the workloads' own densities, cutoffs and skins) and its size.  Operations:

  energy   FField::getE(ener[10]) on the coordinates the engine holds: a full recompute
  frame    a new frame: coordinates uploaded, Verlet list rebuilt, energy recomputed
  delta    the energy change of one trial move, the inner call of a Monte Carlo driver
  drive    MC_metropolis's call sequence on the caller's own arrays: getE, move, getE, restore
  mc       MC_metropolis::run inside the library (on the device, or its host loop)
  host     a batch of chains taken from host buffers, swept once and given back
  sweep    a batch of chains swept on the device, with its running totals read
  total64  the FP64 recompute of every chain's energy (the check of a batch's running totals)
  total32  the mixed-precision recompute of every chain's energy over its lists
"""
import math

import numpy as np
import torch

from mc_cpp_gb300 import systems
from mc_cpp_gb300.engine import BatchChains, FFieldCUDA

KCAL = 418.4               # iu per kcal/mol
COULOMB = 332.0716 * KCAL
RC, RON = 12.0, 10.0
PAIR_FLOPS = 68


def listed():
    return [
        # every Metropolis step of a rigid-water run asks for one of these: a residue's three atoms,
        # some thousand pair terms, so launch and latency are what it costs
        {"name": "delta_water_12288_fp64", "op": "delta", "system": "water", "size": 4096, "prec": "fp64", "cut": "switch"},
        # the small plain workload's energy: 864 argon atoms, the check of a short run's total
        {"name": "energy_argon_864_fp64", "op": "energy", "system": "argon", "size": 864, "prec": "fp64", "cut": "switch"},
        # the middle-sized water box without a cutoff: every pair, as the reference's full mode has it
        {"name": "energy_water_12288_full_fp64", "op": "energy", "system": "water", "size": 4096, "prec": "fp64", "cut": "full"},
        # the large water box in both precisions: energy recomputes of a long run and of analyses
        {"name": "energy_water_100002_fp64", "op": "energy", "system": "water", "size": 33334, "prec": "fp64", "cut": "switch"},
        {"name": "energy_water_100002_mixed", "op": "energy", "system": "water", "size": 33334, "prec": "mixed", "cut": "switch"},
        # a trajectory evaluated frame by frame, with bonded terms and 1-4 pairs: the solvated chain
        {"name": "frame_peptide_18040_fp64", "op": "frame", "system": "peptide", "size": 6000, "prec": "fp64", "cut": "switch"},
        # and a large box, where the list build counts
        {"name": "frame_water_100002_mixed", "op": "frame", "system": "water", "size": 33334, "prec": "mixed", "cut": "switch"},
        # the drop-in use: the reference's Metropolis loop over its own coordinate arrays
        {"name": "drive_water_12288_fp64", "op": "drive", "system": "water", "size": 4096, "prec": "fp64", "cut": "switch", "steps": 50},
        # the library's own run of the small plain workload, translations only (device-resident)
        {"name": "mc_argon_864_fp64", "op": "mc", "system": "argon", "size": 864, "prec": "fp64", "cut": "switch", "steps": 500},
        # the same with translations and rotations of flexible and rigid residues (host loop)
        {"name": "mc_peptide_18040_mixed", "op": "mc", "system": "peptide", "size": 6000, "prec": "mixed", "cut": "switch", "steps": 100},
        # the batched workload end to end: 256 uneven water chains from host memory, one sweep, and back
        {"name": "host_water_256_chains", "op": "host", "system": "water", "chains": 256, "nmin": 512, "nmax": 8192},
        # the FP64 check of a batch's running energies
        {"name": "total64_water_64_chains", "op": "total64", "system": "water", "chains": 64, "nmin": 512, "nmax": 8192},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["delta", "energy", "energy", "energy", "frame", "frame", "drive", "mc", "host", "sweep", "total64", "total32"])
    if op in ("host", "sweep", "total64", "total32"):
        if rng.random() < 0.3:   # atoms: one-atom residues
            return {"op": op, "system": "argon", "chains": _log_int(rng, 4, 256), "nmin": 500, "nmax": rng.randint(501, 2000)}
        nmin = _log_int(rng, 512, 4096)
        return {"op": op, "system": "water", "chains": _log_int(rng, 2, 64), "nmin": nmin, "nmax": _log_int(rng, nmin, 8192)}
    case = {"op": op, "prec": rng.choice(["fp64", "mixed"]), "cut": "switch"}
    system = rng.choice(["argon", "water", "water", "peptide"])
    case["system"] = system
    if op == "mc":
        case["steps"] = rng.randint(20, 200)
        case["size"] = _log_int(rng, 500, 8000) if system == "argon" else _log_int(rng, 512, 8192)
    elif op == "drive":
        case["steps"] = rng.randint(10, 60)
        case["size"] = _log_int(rng, 500, 8000) if system == "argon" else _log_int(rng, 512, 8192)
    else:
        case["size"] = _log_int(rng, 500, 32000) if system == "argon" else _log_int(rng, 512, 33334)
        if op != "frame" and rng.random() < 0.3:
            case["cut"] = "full"
            case["size"] = min(case["size"], 4096)
    return case


# ---- inputs -------------------------------------------------------------------------------------
def _system(case, seed):
    if case["system"] == "argon":
        n = case["size"]
        cells = round((n / 4) ** (1 / 3))
        s = systems.argon_fcc(cells, seed=seed) if 4 * cells ** 3 == n else systems.argon_random(n, 0.0213, seed)
    elif case["system"] == "water":
        s = systems.water_box(case["size"], seed=seed)
    else:   # the box of 6000 waters, scaled to the count
        s = systems.peptide_in_water(40, case["size"], L=56.4 * (case["size"] / 6000) ** (1 / 3) + (0.0 if case["size"] >= 4000 else 1.0),
                                     seed=seed)
    s.cut_mode = case["cut"]
    return s


def _chains(case, seed):
    """The batch's boxes: sizes, densities and temperatures are the case's, positions the seed's."""
    n, lo, hi = case["chains"], case["nmin"], case["nmax"]
    seeds = np.random.default_rng(seed).integers(1, 2 ** 31 - 1, n)
    if case["system"] == "argon":
        rng = np.random.default_rng(5)
        shapes = [(int(rng.integers(lo, hi + 1)), rng.uniform(0.015, 0.025), rng.uniform(90.0, 150.0)) for _ in range(n)]
        return [systems.argon_random(m, rho, int(k), temp) for (m, rho, temp), k in zip(shapes, seeds)]
    return [systems.water_box(m, seed=int(k), temp=temp) for (m, _, temp), k in zip(systems.water_chain_specs(n, lo, hi), seeds)]


def _wrap(v, L):
    return v - L * np.round(v / L)


def _move(s, rng):
    """One trial move of a residue (an atom of argon or of the chain): its atoms and their shift."""
    r = int(rng.integers(1, int(s.resid.max()) + 1))
    idx = np.nonzero(s.resid == r)[0].astype(np.int32)
    if len(idx) > 3:
        idx = idx[int(rng.integers(0, len(idx)))][None]
    return idx, rng.uniform(-0.15, 0.15, 3)


def _shifted(s, seed):
    """The system's coordinates after a short run: every residue displaced a little."""
    rng = np.random.default_rng(seed + 1)
    d = rng.normal(0.0, 0.05, (int(s.resid.max()) + 1, 3))[s.resid]
    return _wrap(s.coords() + d, s.box[0])


def prepare(case, seed):
    st = {"case": case}
    if "chains" in case:
        chains = _chains(case, seed)
        st["batch"] = b = BatchChains(chains, seed=seed)
        if case["op"] == "host":
            n = b.natoms
            xyz = np.concatenate([s.coords() for s in chains]).T
            st["in"] = torch.from_numpy(np.ascontiguousarray(xyz)).pin_memory()
            st["out"] = torch.zeros((3, n), dtype=torch.float64).pin_memory()
        return st
    s = _system(case, seed)
    st["ff"] = FFieldCUDA(s, case["prec"], moves=case["op"] == "mc")
    rng = np.random.default_rng(seed)
    if case["op"] == "delta":
        st["atoms"], shift = _move(s, rng)
        st["new"] = _wrap(s.coords()[st["atoms"]] + shift, s.box[0])
    elif case["op"] == "frame":
        st["xyz"] = _shifted(s, seed)
    elif case["op"] == "drive":
        st["x"], st["y"], st["z"] = s.x.copy(), s.y.copy(), s.z.copy()
        st["L"] = s.box[0]
        st["moves"] = [_move(s, rng) + (float(rng.random()),) for _ in range(case["steps"])]
        st["beta"] = 1.0 / (0.0019872 * s.temp * KCAL)
    elif case["op"] == "mc":
        st["seed"] = seed
    return st


# ---- one pass -----------------------------------------------------------------------------------
def _drive(st):
    ff, x, y, z, L = st["ff"], st["x"], st["y"], st["z"], st["L"]
    e = np.zeros((len(st["moves"]), 2))
    for k, (idx, shift, alpha) in enumerate(st["moves"]):
        e[k, 0] = ff.getE_host(x, y, z)
        old = x[idx], y[idx], z[idx]
        for v, o, d in zip((x, y, z), old, shift):
            v[idx] = _wrap(o + d, L)
        e[k, 1] = ff.getE_host(x, y, z)
        de = e[k, 1] - e[k, 0]
        if not (de <= 0 or alpha < math.exp(-st["beta"] * de)):
            x[idx], y[idx], z[idx] = old
        if (k + 1) % 50 == 0:
            ff.getE_host(x, y, z)
            ff.askListUpdate(k + 1)
    return e, x, y, z


def run(st):
    case = st["case"]
    op = case["op"]
    if op == "energy":
        return st["ff"].getE10()
    if op == "frame":
        st["ff"].setCoords(st["xyz"])
        st["ff"].askListUpdate(0)
        return st["ff"].getE10()
    if op == "delta":
        return st["ff"].delta_e(st["atoms"], st["new"])
    if op == "drive":
        return _drive(st)
    if op == "mc":
        st["seed"] += 1
        _, etot, accepted, _ = st["ff"].metropolis(case["steps"], st["seed"], acceptance="physical", trace=False)
        return etot, accepted, st["ff"].coords()
    b = st["batch"]
    if op == "host":
        accepted, etot = b.run_host(st["in"].numpy(), 1, st["out"].numpy())
        return accepted, etot, st["out"]
    if op == "sweep":
        b.sweep(1)
        return b.stats()
    if op == "total64":
        return b.energy_fp64()
    return b.energy_mixed()


# ---- what a pass cannot do without --------------------------------------------------------------
def _pairs_per_atom(case):
    """Atoms within the cutoff of an atom."""
    rho = {"argon": 0.0213, "water": 3 * 0.0334, "peptide": 3 * 0.0334}[case["system"]]
    return rho * 4.0 / 3.0 * math.pi * RC ** 3


def work(case):
    if "chains" in case:
        if case["system"] == "argon":
            res, apr = case["chains"] * 0.5 * (case["nmin"] + case["nmax"]), 1
        else:
            span = math.log(case["nmax"] / case["nmin"])
            res, apr = case["chains"] * ((case["nmax"] - case["nmin"]) / span if span else case["nmin"]), 3
        n = res * apr
        if case["op"] in ("total64", "total32"):
            return {"bytes": (32 if case["op"] == "total64" else 16) * n, "flops": PAIR_FLOPS * n * _pairs_per_atom(case) / 2}
        moves = {"bytes": 32 * n, "flops": PAIR_FLOPS * n * _pairs_per_atom(case) * 2}
        if case["op"] == "host":
            moves["bytes"] += 48 * n
        return moves
    n = case["size"] if case["system"] == "argon" else 3 * case["size"] + (40 if case["system"] == "peptide" else 0)
    near = _pairs_per_atom(case) if case["cut"] == "switch" else n - 1
    if case["op"] in ("energy", "frame"):
        return {"bytes": (48 if case["op"] == "energy" else 72) * n + 80, "flops": PAIR_FLOPS * n * near / 2}
    moved = 1 if case["system"] == "argon" else 3
    return {"bytes": case.get("steps", 1) * (moved * near + 1) * 48, "flops": case.get("steps", 1) * 2 * PAIR_FLOPS * moved * near}


# ---- the same numbers in 64 bits ----------------------------------------------------------------
class _Box:
    """One box's coordinates and parameters as FP64 tensors; molecules exclude their own pairs."""

    def __init__(self, s, xyz):
        dev = "cuda" if torch.cuda.is_available() else "cpu"

        def t(a):
            return torch.as_tensor(np.asarray(a), dtype=torch.float64, device=dev)
        self.xyz, self.q, self.sig, self.L, self.switch = t(xyz), t(s.q), t(s.sig), float(s.box[0]), s.cut_mode == "switch"
        self.eps = torch.sqrt(t(s.eps) * KCAL)
        self.mol = torch.as_tensor(np.asarray(s.resid), device=dev)

    def between(self, i, xyz_i):
        """Sums (elec, vdw) of atoms i, at xyz_i, with every other atom."""
        d = [xyz_i[:, k, None] - self.xyz[None, :, k] for k in range(3)]
        r2 = sum((v - self.L * torch.round(v / self.L)) ** 2 for v in d)
        keep = self.mol[i][:, None] != self.mol[None, :]
        if self.switch:
            keep &= r2 <= RC * RC
        a, b = torch.nonzero(keep, as_tuple=True)
        r2 = r2[a, b]
        a = i[a]
        elec = self.q[a] * self.q[b] / torch.sqrt(r2)
        x6 = ((self.sig[a] + self.sig[b]) ** 2 / r2) ** 3
        vdw = self.eps[a] * self.eps[b] * (x6 * x6 - x6)
        if self.switch:
            u = r2.clamp(min=RON * RON)
            f = (RC * RC - u) ** 2 * (RC * RC + 2 * u - 3 * RON * RON) / (RC * RC - RON * RON) ** 3
            elec, vdw = elec * f, vdw * f
        return COULOMB * elec.sum().item(), 4 * vdw.sum().item()

    def total(self):
        n = len(self.xyz)
        rows = max(1, 40_000_000 // n)
        parts = []
        for b in range(0, n, rows):
            i = torch.arange(b, min(n, b + rows), device=self.xyz.device)
            parts.append(self.between(i, self.xyz[i]))
        return [0.5 * math.fsum(p[k] for p in parts) for k in (0, 1)]


def _bonded(s, xyz):
    """Harmonic bonds and angles (all that water has)."""
    L = s.box[0]
    if not len(s.bonds):
        return 0.0, 0.0
    d = _wrap(xyz[s.bonds[:, 0]] - xyz[s.bonds[:, 1]], L)
    r = np.sqrt((d * d).sum(1))
    bond = math.fsum(0.5 * s.bond_k * KCAL * (r - s.bond_r0) ** 2)
    u, v = (_wrap(xyz[s.angles[:, k]] - xyz[s.angles[:, 1]], L) for k in (0, 2))
    c = (u * v).sum(1) / np.sqrt((u * u).sum(1) * (v * v).sum(1))
    angle = math.fsum(0.5 * s.angle_k * KCAL * (np.arccos(c) - s.angle_theta0 * np.pi / 180) ** 2)
    return bond, angle


def exact(case, seed):
    if case["system"] == "peptide" or case["op"] in ("drive", "mc", "host", "sweep"):
        return None   # 1-4 and exclusion rules beyond plain sums, and runs of many decisions
    if "chains" in case:
        return np.array([sum(_Box(s, s.coords()).total()) for s in _chains(case, seed)])
    s = _system(case, seed)
    if case["op"] == "delta":
        box = _Box(s, s.coords())
        idx, shift = _move(s, np.random.default_rng(seed))
        new = _wrap(s.coords()[idx] + shift, s.box[0])
        i = torch.as_tensor(idx.astype(np.int64), device=box.xyz.device)
        e = [sum(box.between(i, torch.as_tensor(p, device=box.xyz.device))) for p in (new, s.coords()[idx])]
        moved = s.coords()
        moved[idx] = new
        return e[0] - e[1] + sum(_bonded(s, moved)) - sum(_bonded(s, s.coords()))
    xyz = _shifted(s, seed) if case["op"] == "frame" else s.coords()
    elec, vdw = _Box(s, xyz).total()
    bond, angle = _bonded(s, xyz)
    tot = elec + vdw + bond + angle
    return np.array([tot, tot, 0.0, elec, vdw, bond, angle, 0.0, 0.0, 0.0])
