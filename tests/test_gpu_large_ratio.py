"""Walkers next to a node of the ground determinant, where excited determinants exceed it
by factors above the kernels' lines (256, 4096): the local energy evaluates them a second
time, the gradient, drift, HMC and adjoint kernels sum over explicit determinants. Compared
with the same wave function given as an explicit list of configurations, whose kernels
factor every determinant."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def columns(tables, spin, n):
    """Orbitals of each unique determinant of an excitation table, position by position."""
    nv, rows = tables.max_orb[spin] - n, []
    for order, i0, i1, i2, _ in tables.t["det_table%d" % spin].cpu().numpy().reshape(-1, 5):
        row = list(range(n))
        if order >= 1:
            row[i0 // nv] = n + i0 % nv
        if order == 2:
            row[i2 // nv] = n + i1 % nv
        rows.append(row)
    return torch.as_tensor(rows)


@pytest.fixture(scope="module")
def waves():
    """(excitation-mode wave function, the explicit one, walkers with ratios of 5e3 to 2e5,
    their ratios)."""
    from qmctorch_gb300.scf import Molecule
    from qmctorch_gb300.serving import seeded_positions
    from qmctorch_gb300.wavefunction import SlaterJastrow
    torch.set_default_dtype(torch.float64)
    mol = Molecule("O 0 0 0.1173; H 0 0.7572 -0.4692; H 0 -0.7572 -0.4692", unit="angs",
                   basis="cc-pvdz", calculator="huckel")
    wf = SlaterJastrow(mol, configs="single_double(4,4)", cuda=True)
    tab = wf.pool._tables
    cfg = tuple(columns(tab, s, 5)[tab.t["cfg_det%d" % s].cpu().long()] for s in range(2))
    ex = SlaterJastrow(mol, configs=cfg, cuda=True)
    weight = torch.as_tensor(np.random.default_rng(5).uniform(0.2, 1.0, size=(1, wf.nci))).cuda()
    for w in (wf, ex):
        w.fc.weight.data = weight.clone()
    x = torch.as_tensor(seeded_positions(mol, 200_000, 9), device="cuda")
    with torch.no_grad():
        mo = torch.cat([wf.mo(wf.ao(c)) for c in x.split(20_000)])
        ratio = 0
        for s in range(2):
            m = mo[:, 5 * s:5 * s + 5]
            d = torch.stack([torch.linalg.det(m[:, :, c]) for c in columns(tab, s, 5).cuda()], 1)
            ratio = torch.maximum(d.abs().amax(1) / d[:, 0].abs(), torch.as_tensor(ratio).cuda())
    keep = (ratio > 5e3) & (ratio < 2e5)
    assert int(keep.sum()) > 10
    return wf, ex, x[keep][:64].contiguous(), ratio[keep][:64]


def test_local_energy(waves):
    wf, ex, x, ratio = waves
    other = torch.as_tensor(np.random.default_rng(1).normal(size=(40, 30))).cuda() + x[:1]
    with torch.no_grad():
        got = wf.local_energy(torch.cat([other, x]))[40:].reshape(-1)
        assert torch.equal(got, wf.local_energy(x).reshape(-1))  # whatever else the block holds
        want = ex.local_energy(x).reshape(-1)
    # rounding (1e-16), amplified by the ratio's square and a matrix of condition 1e3
    assert ((got - want).abs() <= 1e-13 * ratio ** 2 * (1 + want.abs())).all()


def test_gradients(waves):
    wf, ex, x, _ = waves
    got, want = wf.gradients(x), ex.gradients(x)
    scale = want.abs().amax(1, keepdim=True)
    assert ((got - want) / scale).abs().max() < 1e-10  # both sum the same determinants


@pytest.mark.parametrize("kind", ["psi", "eloc"])
def test_adjoints(waves, kind):
    wf, ex, x, _ = waves
    grads = []
    for w in (wf, ex):
        for p in w.parameters():
            p.grad = None
        (w(x) if kind == "psi" else w.local_energy(x)).sum().backward()
        grads.append([w.ao.bas_exp.grad, w.mo.mo_modifier.grad, w.fc.weight.grad,
                      w.jastrow.jastrow_kernel.weight.grad])
    for got, want in zip(*grads):
        assert (got - want).abs().max() <= 1e-9 * want.abs().max()


@pytest.mark.parametrize("kind", ["drift", "hmc"])
def test_samplers(waves, kind):
    """Short moves from these walkers: the proposals stay next to the node."""
    from qmctorch_gb300.sampler import GeneralizedMetropolis, Hamiltonian
    wf, ex, x, _ = waves
    out = []
    for w in (wf, ex):
        torch.manual_seed(3)
        common = dict(nwalkers=len(x), nstep=3, ntherm=0, nelec=10, ndim=3, cuda=True, rng="torch")
        s = (GeneralizedMetropolis(step_size=1e-7, **common) if kind == "drift"
             else Hamiltonian(step_size=1e-6, L=2, **common))
        out.append(s(w.pdf, pos=x.clone(), with_tqdm=False).detach())
    assert torch.isfinite(out[0]).all()
    assert (out[0] - out[1]).abs().max() < 1e-8
