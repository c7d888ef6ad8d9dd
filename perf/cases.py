"""Measured workloads of the framework: what a variational Monte Carlo user has it do,
through the public entry points, from the smallest calls to the largest.

Molecules, bases and configuration sets are those of the benchmark and the tests: H2, LiH
and linear H_n chains in sto-3g, H2O in cc-pVDZ with single_double(4,4), C6H6 in cc-pVDZ
with its ground-state determinant. Walkers are seeded Gaussians around the nuclei, as there,
equilibrated where local energies are asked for.
"""
import functools
import math

import numpy as np
import torch

from qmctorch_gb300.sampler import GeneralizedMetropolis, Hamiltonian, Metropolis
from qmctorch_gb300.scf import Molecule
from qmctorch_gb300.solver import Solver
from qmctorch_gb300.wavefunction import SlaterJastrow
from qmctorch_gb300.wavefunction.jastrows import (JastrowFactorElectronElectron,
                                                  JastrowFactorElectronNuclei)

torch.set_default_dtype(torch.float64)

# molecule -> (geometry in angstrom, basis, calculator, configurations)
MOLECULES = {
    "H2": ("H 0 0 -0.37; H 0 0 0.37", "sto-3g", "pyscf", "ground_state"),
    "LiH": ("Li 0 0 0; H 0 0 1.595", "sto-3g", "pyscf", "cas(2,2)"),
    "H2O": ("O 0 0 0.1173; H 0 0.7572 -0.4692; H 0 -0.7572 -0.4692", "cc-pvdz", "pyscf",
            "single_double(4,4)"),
    "C6H6": ("C 1.39 0 0; C 0.695 1.20377 0; C -0.695 1.20377 0; C -1.39 0 0; "
             "C -0.695 -1.20377 0; C 0.695 -1.20377 0; H 2.48 0 0; H 1.24 2.14774 0; "
             "H -1.24 2.14774 0; H -2.48 0 0; H -1.24 -2.14774 0; H 1.24 -2.14774 0",
             "cc-pvdz", "huckel", "ground_state"),
}


def listed():
    """Twelve cases. ``en``: the electron-nucleus Jastrow factor beside the electron-electron
    one; ``precision``: the method of the fused kernels ("fp64" is the default of a program in
    double precision, "mixed" the fast method)."""
    return [
        # a single point on the smallest molecule: sampling, local energies and statistics of
        # a few walkers, where launches and the host path count
        {"name": "h2_single_point", "kind": "single_point", "mol": "H2", "precision": "fp64",
         "en": False, "nw": 256, "nstep": 50},
        # the benchmark's headline: all-electron moves of many walkers, the fast method
        {"name": "h2o_metropolis_mixed", "kind": "metropolis", "mol": "H2O",
         "precision": "mixed", "en": False, "nw": 16384, "nstep": 100},
        # the default method between two optimisation epochs (25 update steps), a ragged
        # number of walkers
        {"name": "h2o_metropolis_fp64", "kind": "metropolis", "mol": "H2O",
         "precision": "fp64", "en": False, "nw": 5001, "nstep": 25},
        # a long chain in the default method, as a request of the serving loop has it
        {"name": "h24_metropolis_fp64", "kind": "metropolis", "mol": "H24",
         "precision": "fp64", "en": False, "nw": 2048, "nstep": 50},
        # sweeps of single-electron moves of the largest molecule (Sherman-Morrison)
        {"name": "c6h6_sweep_mixed", "kind": "sweep", "mol": "C6H6", "precision": "mixed",
         "en": False, "nw": 16384, "nstep": 2},
        # local energies of all kept samples of a single point, the default method
        {"name": "h2o_eloc_fp64", "kind": "eloc", "mol": "H2O", "precision": "fp64",
         "en": False, "nw": 50003},
        # local energies of the largest molecule, the fast method on single-precision walkers
        {"name": "c6h6_eloc_mixed", "kind": "eloc", "mol": "C6H6", "precision": "mixed",
         "en": False, "nw": 16384},
        # one optimisation step with the default (manual) gradient: E_L and psi forward, psi
        # backward to every parameter; the reference's small CAS configuration
        {"name": "lih_manual_step", "kind": "step", "grad": "manual", "mol": "LiH",
         "precision": "fp64", "en": False, "nw": 8192},
        # the same through the local energy itself, multi-determinant H2O
        {"name": "h2o_auto_step", "kind": "step", "grad": "auto", "mol": "H2O",
         "precision": "fp64", "en": False, "nw": 4000},
        # the drift-diffusion sampler (position gradients at every proposal)
        {"name": "h2o_drift", "kind": "drift", "mol": "H2O", "precision": "fp64", "en": False,
         "nw": 8192, "nstep": 50},
        # Hamiltonian Monte Carlo: full position gradients along leapfrog trajectories
        {"name": "h2o_hmc", "kind": "hmc", "mol": "H2O", "precision": "fp64", "en": False,
         "nw": 8192, "nstep": 2, "traj": 5},
        # the layers one by one, as a program that works on orbitals calls them: atomic
        # orbitals, molecular orbitals, Slater determinants, Jastrow factor
        {"name": "h2o_layers", "kind": "layers", "mol": "H2O", "precision": "fp64",
         "en": False, "nw": 16384},
    ]


# walkers (and steps) of the drawn cases, kind -> (molecules, precisions, (low, high) per size)
RANGES = {
    "single_point": (("H2", "LiH"), ("fp64", "mixed"), {"nw": (64, 2048), "nstep": (20, 100)}),
    "metropolis": (("LiH", "H2O", "H8", "H16", "H24"), ("fp64", "mixed"),
                   {"nw": (500, 8192), "nstep": (10, 50)}),
    "sweep": (("C6H6", "H16", "H24"), ("fp64", "mixed"), {"nw": (256, 4096), "nstep": (1, 2)}),
    "eloc": (("LiH", "H2O", "H16", "C6H6"), ("fp64", "mixed"), {"nw": (1000, 16384)}),
    "step": (("H2", "LiH", "H2O"), ("fp64",), {"nw": (500, 16384)}),
    "drift": (("H2", "LiH", "H2O"), ("fp64",), {"nw": (500, 8192), "nstep": (10, 50)}),
    "hmc": (("H2", "LiH", "H2O"), ("fp64",), {"nw": (500, 8192), "nstep": (1, 2),
                                              "traj": (3, 5)}),
    "layers": (("LiH", "H2O", "H16"), ("fp64",), {"nw": (500, 16384)}),
}


def draw(rng):
    """One more case of the listed kinds: another molecule, precision, Jastrow factor, size."""
    kind = rng.choice(sorted(RANGES))
    mols, precisions, sizes = RANGES[kind]
    case = {"kind": kind, "mol": rng.choice(mols), "precision": rng.choice(precisions),
            "en": kind != "layers" and rng.random() < 0.3}
    if kind == "step":
        case["grad"] = rng.choice(("manual", "auto"))
    for key, (low, high) in sizes.items():
        case[key] = int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))
    return case


@functools.lru_cache(maxsize=None)
def _molecule(name):
    if name in MOLECULES:
        atoms, basis, calculator, configs = MOLECULES[name]
    else:  # a linear chain of hydrogen atoms, 0.95 angstrom apart
        atoms = "; ".join("H 0 0 %.10f" % (0.95 * i) for i in range(int(name[1:])))
        basis, calculator, configs = "sto-3g", "huckel", "ground_state"
    return Molecule(atoms, unit="angs", basis=basis, calculator=calculator), configs


def _wavefunction(case, cuda=True):
    mol, configs = _molecule(case["mol"])
    jastrow = "default"
    if case["en"]:
        jastrow = [JastrowFactorElectronElectron(mol), JastrowFactorElectronNuclei(mol)]
    wf = SlaterJastrow(mol, jastrow=jastrow, configs=configs, cuda=cuda,
                       precision=case["precision"])
    # CI weights as an optimisation has them: every configuration takes part
    weight = np.random.default_rng(7).uniform(size=wf.nci)
    wf.fc.weight.data = torch.as_tensor(weight, device=wf.fc.weight.device).reshape(1, -1)
    return wf


def _positions(case, seed):
    mol, _ = _molecule(case["mol"])
    g = torch.Generator().manual_seed(int(seed))
    centers = np.repeat(np.asarray(mol.atom_coords), mol.atomic_nelec, axis=0)[: mol.nelec]
    x = torch.as_tensor(centers).unsqueeze(0) + torch.randn((case["nw"], mol.nelec, 3),
                                                            generator=g)
    x = x.reshape(case["nw"], -1).cuda()
    if case["kind"] not in ("eloc", "step"):
        return x
    # local energies are asked for at walkers that follow psi^2 (elsewhere their tail at the
    # nodes outweighs everything): some steps of the default method, in sweeps of
    # single-electron moves where there is one determinant
    sweep = case["mol"] in ("C6H6", "H16")
    sampler = Metropolis(nwalkers=case["nw"], nstep=20 if sweep else 40, step_size=0.2, ntherm=-1,
                         nelec=mol.nelec, init=mol.domain("atomic"), cuda=True,
                         move={"type": "all-elec-iter" if sweep else "all-elec",
                               "proba": "normal"}, seed=101 + int(seed))
    sampler(_wavefunction(dict(case, precision="fp64")).pdf, pos=x, with_tqdm=False)
    # the fast method's local energies are asked for with single-precision walkers
    return x.float() if case["precision"] == "mixed" else x


def prepare(case, seed):
    """The wave function, the sampler or solver of the call, and the walkers."""
    wf = _wavefunction(case)
    mol, kind = wf.mol, case["kind"]
    state = {"kind": kind, "wf": wf, "seed": int(seed)}
    common = {"nwalkers": case["nw"], "nstep": case.get("nstep", 1), "nelec": mol.nelec,
              "ndim": 3, "cuda": True, "seed": 1 + int(seed)}
    if kind == "single_point":
        sampler = Metropolis(step_size=0.2, ntherm=case["nstep"] // 2, ndecor=5,
                             init=mol.domain("uniform"), **common)
        state["solver"] = Solver(wf=wf, sampler=sampler)
        return state
    state["x"] = _positions(case, seed)
    if kind in ("metropolis", "sweep"):
        move = "all-elec" if kind == "metropolis" else "all-elec-iter"
        state["sampler"] = Metropolis(step_size=0.2 if kind == "metropolis" else 0.1, ntherm=-1,
                                      move={"type": move, "proba": "normal"},
                                      init=mol.domain("atomic"), **common)
    elif kind == "drift":
        state["sampler"] = GeneralizedMetropolis(step_size=0.05, ntherm=-1, **common)
    elif kind == "hmc":
        state["sampler"] = Hamiltonian(step_size=0.02, L=case["traj"], ntherm=-1, **common)
    elif kind == "step":
        sampler = Metropolis(init=mol.domain("atomic"), **common)
        opt = torch.optim.Adam(wf.parameters(), lr=1e-3)
        state["solver"] = Solver(wf=wf, sampler=sampler, optimizer=opt)
        state["solver"].configure(loss="energy", grad=case["grad"])
    return state


def run(state):
    """One pass through the public entry points."""
    wf, kind = state["wf"], state["kind"]
    if kind == "single_point":
        torch.manual_seed(state["seed"])  # the walkers' initial positions
        obs = state["solver"].single_point(with_tqdm=False)
        return {"pos": obs.pos, "local_energy": obs.local_energy, "energy": obs.energy,
                "variance": obs.variance, "error": obs.error}
    x = state["x"]
    if kind in ("metropolis", "sweep", "drift", "hmc"):
        # the samplers move the walkers that they are given
        return state["sampler"](wf.pdf, pos=x.clone(), with_tqdm=False)
    if kind == "eloc":
        with torch.no_grad():
            return wf.local_energy(x)
    if kind == "step":
        solver = state["solver"]
        solver.opt.zero_grad()
        loss, eloc = solver.evaluate_gradient(x)
        grads = {name: p.grad for name, p in wf.named_parameters() if p.grad is not None}
        return {"loss": loss, "local_energy": eloc, "grads": grads}
    with torch.no_grad():
        ao = wf.ao(x)
        mo = wf.mo(ao)
        return {"ao": ao, "mo": mo, "dets": wf.pool(mo), "jastrow": wf.jastrow(x)}


def work(case):
    """Bytes in and out, and the operations of the formulas (an exponential counts as ten)."""
    wf = _wavefunction(case, cuda=False)
    mol, basis, nw, kind = wf.mol, wf.ao._basis, case["nw"], case["kind"]
    ne, nao, nmu = mol.nelec, wf.ao.norb, wf.highest_occ_mo
    nexp = len({(int(a), float(e)) for a, e in zip(
        np.repeat(np.arange(mol.natom), basis.nshells), basis.bas_exp)})
    nent = len(basis.bas_exp)
    row_ao = 10 * nexp + 2 * nent + 3 * nao          # the AO values of one electron
    lu = sum(2 * n ** 3 / 3 + 2 * n * n * (nmu - n) for n in (mol.nup, mol.ndown))
    pairs = 14 * (ne * (ne - 1) / 2 + (ne * mol.natom if case["en"] else 0))
    psi = ne * (row_ao + 2 * nao * nmu) + pairs + lu + 3 * wf.nci
    grad = ne * (row_ao + 6 * nent + 9 * nao + 8 * nao * nmu) + 3 * pairs + 3 * lu + 3 * wf.nci
    eloc = ne * (row_ao + 4 * nent + 12 * nao + 6 * nao * nmu) + 3 * pairs + 4 * lu + 6 * wf.nci
    pos = 8 * 3 * ne * nw
    if kind == "single_point":
        kept = len(range(case["nstep"] // 2, case["nstep"], 5))
        return {"bytes": pos * (1 + kept) + 8 * nw * kept,
                "flops": nw * (case["nstep"] * psi + kept * eloc)}
    if kind == "metropolis":
        return {"bytes": 3 * pos, "flops": nw * case["nstep"] * psi}
    if kind == "sweep":
        n = mol.nup
        move = row_ao + 2 * nao * n + 2 * n * n + 28 * ne + n * n
        return {"bytes": 3 * pos, "flops": nw * case["nstep"] * ne * move}
    if kind == "drift":
        n = mol.nup
        move = row_ao + 6 * nent + 9 * nao + 8 * nao * nmu + 42 * ne + lu / 2 + 6 * n * nmu
        return {"bytes": 3 * pos, "flops": nw * (grad + case["nstep"] * move)}
    if kind == "hmc":
        return {"bytes": 3 * pos, "flops": nw * case["nstep"] * (case["traj"] + 1) * grad}
    if kind == "eloc":
        return {"bytes": pos * (1 if case["precision"] == "fp64" else 0.5) + 8 * nw,
                "flops": nw * eloc}
    if kind == "step":
        params = 8 * (nent + nao * wf.mo.mo_scf.shape[1] + wf.nci + 2)
        back = 2 * (psi if case["grad"] == "manual" else eloc)
        return {"bytes": 2 * pos + 16 * nw + params,
                "flops": nw * (eloc + back + (psi if case["grad"] == "manual" else 0))}
    nmo = wf.mo.mo_scf.shape[1]
    return {"bytes": pos + 8 * nw * (ne * (nao + nmo) + wf.nci + 1),
            "flops": nw * (ne * (row_ao + 2 * nao * nmo) + pairs + lu + 3 * wf.nci)}


# ----------------------------------------------------------------------------
# the same quantities in plain torch, 64 bits
# ----------------------------------------------------------------------------
class _Plain:
    """The Slater-Jastrow wave function from its definition: contracted cartesian Gaussians,
    one determinant per unique configuration and spin, Pade factors. ``theta`` holds the
    parameters (leaves, so that autograd gives their gradients)."""

    def __init__(self, case):
        wf = _wavefunction(case, cuda=False)
        dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
        t = lambda v, dt=torch.float64: torch.as_tensor(np.asarray(v)).to(dev, dt)  # noqa: E731
        b, mol = wf.ao._basis, wf.mol
        self.dev, self.nup, self.ne, self.natom = dev, mol.nup, mol.nelec, mol.natom
        self.atoms, self.charge = t(mol.atom_coords), t(mol.atomic_number)
        self.entry_atom = t(np.repeat(np.arange(mol.natom), b.nshells), torch.long)
        k = np.stack([b.bas_kx, b.bas_ky, b.bas_kz], 1).astype(int)
        self.k, self.index = t(k), t(b.index_ctr, torch.long)
        # cartesian Gaussian norms from the basis' exponents (constants), times the coefficients
        odd = {0: 1.0, 1: 1.0, 2: 3.0}
        norm = (2 * b.bas_exp / np.pi) ** 0.75
        for c in range(3):
            norm = norm * (4 * b.bas_exp) ** (k[:, c] / 2) / np.sqrt([odd[v] for v in k[:, c]])
        self.weight = t(norm * b.bas_coeffs)
        self.contract = torch.zeros((len(b.bas_exp), wf.ao.norb), device=dev)
        self.contract[torch.arange(len(b.bas_exp), device=dev), self.index] = 1.0
        self.scf, self.nmu = wf.mo.mo_scf.detach().to(dev).double(), wf.highest_occ_mo
        self.theta = {n: p.detach().to(dev).double().requires_grad_(True)
                      for n, p in wf.named_parameters() if n != "ao.atom_coords"}
        jw = sorted(n for n in self.theta if n.startswith("jastrow"))
        self.wee, self.wen = jw[0], (jw[1] if case["en"] else None)
        tab = wf.pool._tables
        self.cfg = [tab.t["cfg_det%d" % s].long().to(dev) for s in range(2)]
        self.cols = [self._columns(tab, s, (mol.nup, mol.ndown)[s]).to(dev) for s in range(2)]
        self.vnn = sum(mol.atomic_number[i] * mol.atomic_number[j]
                       / float(np.linalg.norm(np.subtract(mol.atom_coords[i], mol.atom_coords[j])))
                       for i in range(mol.natom) for j in range(i))

    @staticmethod
    def _columns(tab, spin, n):
        """Orbitals of each unique determinant, position by position."""
        raw = tab.t["det_table%d" % spin].cpu().numpy()
        if tab.explicit:
            return torch.as_tensor(raw.reshape(-1, n)).long()
        nv, rows = tab.max_orb[spin] - n, []
        for order, i0, i1, i2, _ in raw.reshape(-1, 5):
            row = list(range(n))
            if order >= 1:
                row[i0 // nv] = n + i0 % nv
            if order == 2:
                row[i2 // nv] = n + i1 % nv
            rows.append(row)
        return torch.as_tensor(rows).long()

    def orbitals(self, x, derivatives):
        """AO values (and gradients, Laplacians) [walker, electron, ao]."""
        d = x.view(len(x), self.ne, 1, 3) - self.atoms
        d = d[:, :, self.entry_atom]
        r2, a = (d * d).sum(-1), self.theta["ao.bas_exp"]
        power = lambda k: torch.where(k <= 0, torch.ones_like(d),  # noqa: E731
                                      torch.where(k == 1, d, d * d))
        e = self.weight * torch.exp(-a * r2)
        p0 = power(self.k)
        poly = p0.prod(-1)
        val = (e * poly) @ self.contract
        if not derivatives:
            return val
        p1 = self.k * power(self.k - 1)
        p2 = self.k * (self.k - 1) * power(self.k - 2)
        grads, lap = [], 0
        for c in range(3):
            other = p0[..., (c + 1) % 3] * p0[..., (c + 2) % 3]
            grads.append((e * (p1[..., c] * other - 2 * a * d[..., c] * poly)) @ self.contract)
            lap = lap + p2[..., c] * other
        degree = self.k.sum(-1)
        lap = e * (lap - 4 * a * degree * poly + poly * (4 * a * a * r2 - 6 * a))
        return val, grads, lap @ self.contract

    def jastrow(self, x, derivatives):
        """log J (and its gradient [walker, electron, 3] and Laplacian [walker, electron])."""
        r = x.view(len(x), self.ne, 3)
        d = r.unsqueeze(2) - r.unsqueeze(1)
        eye = torch.eye(self.ne, device=self.dev)
        dist = ((d * d).sum(-1) + eye).sqrt()
        spin = torch.arange(self.ne, device=self.dev) < self.nup
        w0 = torch.where(spin.unsqueeze(0) == spin.unsqueeze(1), 0.25, 0.5) * (1 - eye)
        terms = [(d, dist, w0, self.theta[self.wee], 0.5)]
        if self.wen is not None:
            da = r.unsqueeze(2) - self.atoms
            terms.append((da, da.norm(dim=-1), torch.ones(1, device=self.dev),
                          self.theta[self.wen], 1.0))
        u, g, lap = 0, 0, 0
        for d, dist, w0, w, half in terms:
            s = 1 / (1 + w * dist)
            u = u + half * (w0 * dist * s).sum((1, 2))
            if derivatives:
                k1 = w0 * s * s
                g = g + ((k1 / dist).unsqueeze(-1) * d).sum(2)
                lap = lap + (2 * k1 / dist - 2 * w * k1 * s).sum(2)
        return (u, g, lap) if derivatives else u

    def spins(self, m):
        """Rows of the up and the down electrons."""
        return m[:, : self.nup], m[:, self.nup:]

    def matrices(self, rows, s):
        """[walker, determinant, electron, orbital] of spin s from the rows of its electrons."""
        return rows[:, :, self.cols[s]].permute(0, 2, 1, 3)

    def psi(self, x):
        mo = self.orbitals(x, False) @ self.mos()
        det = [torch.linalg.det(self.matrices(m, s)) for s, m in enumerate(self.spins(mo))]
        c = self.theta["fc.weight"].reshape(-1)
        return torch.exp(self.jastrow(x, False)) * (det[0][:, self.cfg[0]]
                                                    * det[1][:, self.cfg[1]] * c).sum(1)

    def mos(self):
        return (self.scf * self.theta["mo.mo_modifier"])[:, : self.nmu]

    def eloc(self, x):
        val, grads, lap = self.orbitals(x, True)
        w = self.mos()
        _, g, lj = self.jastrow(x, True)
        a = val @ w
        b = lap @ w + (lj + (g * g).sum(-1)).unsqueeze(-1) * a
        for c in range(3):
            b = b + 2 * g[..., c: c + 1] * (grads[c] @ w)
        det, tr = [], []
        for s, (ra, rb) in enumerate(zip(self.spins(a), self.spins(-0.5 * b))):
            ma = self.matrices(ra, s)
            det.append(torch.linalg.det(ma)[:, self.cfg[s]])
            trace = torch.linalg.solve(ma, self.matrices(rb, s)).diagonal(dim1=-2, dim2=-1)
            tr.append(trace.sum(-1)[:, self.cfg[s]])
        cd = self.theta["fc.weight"].reshape(-1) * det[0] * det[1]
        kin = (cd * (tr[0] + tr[1])).sum(1) / cd.sum(1)
        r = x.view(len(x), self.ne, 3)
        ven = -(self.charge / (r.unsqueeze(2) - self.atoms).norm(dim=-1)).sum((1, 2))
        d = r.unsqueeze(2) - r.unsqueeze(1)
        i, j = torch.triu_indices(self.ne, self.ne, 1)
        return kin + ven + (1 / d[:, i, j].norm(dim=-1)).sum(1) + self.vnn


def exact(case, seed):
    """What ``run`` returns, in plain torch: local energies, gradients, layers; chains of
    random moves have no such value."""
    kind, nw = case["kind"], case["nw"]
    if kind not in ("eloc", "step", "layers"):
        return None
    plain, x = _Plain(case), _positions(case, seed).double()
    chunks = x.split(250 if case["mol"] == "C6H6" else 1000)
    with torch.no_grad():
        if kind == "eloc":
            return torch.cat([plain.eloc(c) for c in chunks]).reshape(-1, 1)
        if kind == "layers":
            ao = torch.cat([plain.orbitals(c, False) for c in chunks])
            mo = ao @ (plain.scf * plain.theta["mo.mo_modifier"])
            dets = 1
            for s, rows in enumerate(plain.spins(mo)):
                one = torch.cat([torch.linalg.det(plain.matrices(m, s))
                                 for m in rows.split(1000)])
                dets = dets * one[:, plain.cfg[s]]
            jas = torch.cat([torch.exp(plain.jastrow(c, False)) for c in chunks])
            return {"ao": ao, "mo": mo, "dets": dets, "jastrow": jas.reshape(-1, 1)}
        eloc = torch.cat([plain.eloc(c) for c in chunks])
        mean = eloc.mean()
    at = 0
    for c in chunks:
        el = eloc[at: at + len(c)]
        at += len(c)
        if case["grad"] == "manual":
            psi = plain.psi(c)
            (psi * (2 / nw * (el - mean) / psi.detach())).sum().backward()
        else:
            (plain.eloc(c).sum() / nw).backward()
    grads = {n: p.grad for n, p in plain.theta.items() if p.grad is not None}
    return {"loss": mean, "local_energy": eloc.reshape(-1, 1), "grads": grads}
