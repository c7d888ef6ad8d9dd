"""Gradients, adjoints, drift and HMC with 1 to 7 electrons per spin: excitation mode
(factors of the ground determinant) against the same configurations as explicit lists (sums
over determinants: in a warp's registers up to five electrons, a chain per thread beyond),
at walker counts that leave blocks and warps partly empty."""
import numpy as np
import pytest
import torch

from tests.test_gpu_large_ratio import columns

pytestmark = pytest.mark.gpu

def chain(n):
    return "; ".join("H 0 0 %g" % (0.95 * i) for i in range(2 * n))


MOLECULES = {  # electrons per spin -> geometry, configurations
    1: (chain(1), "single_double(2,2)"),
    2: ("Li 0 0 0; H 0 0 1.595", "single_double(2,4)"),
    3: (chain(3), "single_double(4,4)"),
    4: (chain(4), "single_double(4,4)"),
    5: ("O 0 0 0.1173; H 0 0.7572 -0.4692; H 0 -0.7572 -0.4692", "single_double(4,4)"),
    7: (chain(7), "single_double(4,4)"),
}


def waves(n):
    from qmctorch_gb300.scf import Molecule
    from qmctorch_gb300.wavefunction import SlaterJastrow
    torch.set_default_dtype(torch.float64)
    atoms, configs = MOLECULES[n]
    mol = Molecule(atoms, unit="angs", basis="sto-3g", calculator="huckel")
    wf = SlaterJastrow(mol, configs=configs, cuda=True)
    assert mol.nup == n
    tab = wf.pool._tables
    cfg = tuple(columns(tab, s, n)[tab.t["cfg_det%d" % s].cpu().long()] for s in range(2))
    ex = SlaterJastrow(mol, configs=cfg, cuda=True)
    weight = torch.as_tensor(np.random.default_rng(n).uniform(0.2, 1.0, size=(1, wf.nci))).cuda()
    for w in (wf, ex):
        w.fc.weight.data = weight.clone()
    return mol, wf, ex


@pytest.mark.parametrize("nw", [1, 33, 150])
@pytest.mark.parametrize("n", sorted(MOLECULES))
def test_modes_agree(n, nw):
    from qmctorch_gb300.sampler import GeneralizedMetropolis, Hamiltonian
    from qmctorch_gb300.serving import seeded_positions
    mol, wf, ex = waves(n)
    x = torch.as_tensor(seeded_positions(mol, nw, 4), device="cuda")
    # rounding amplified by the matrices' condition (1e4) and the excitation ratios
    got, want = wf.gradients(x), ex.gradients(x)
    assert ((got - want).abs() <= 1e-8 * want.abs().amax(1, keepdim=True)).all()
    for kind in ("psi", "eloc"):
        grads = []
        for w in (wf, ex):
            for p in w.parameters():
                p.grad = None
            (w(x) if kind == "psi" else w.local_energy(x)).sum().backward()
            grads.append([w.ao.bas_exp.grad, w.mo.mo_modifier.grad, w.fc.weight.grad,
                          w.jastrow.jastrow_kernel.weight.grad])
        for a, b in zip(*grads):
            assert (a - b).abs().max() <= 1e-8 * max(float(b.abs().max()), 1e-6)
    common = dict(nwalkers=nw, nstep=3, ntherm=0, nelec=mol.nelec, ndim=3, cuda=True, rng="torch")
    for make in (lambda: GeneralizedMetropolis(step_size=1e-4, **common),
                 lambda: Hamiltonian(step_size=1e-4, L=2, **common)):
        out = []
        for w in (wf, ex):
            torch.manual_seed(3)
            out.append(make()(w.pdf, pos=x.clone(), with_tqdm=False).detach())
        assert torch.isfinite(out[0]).all()
        assert (out[0] - out[1]).abs().max() < 1e-7
