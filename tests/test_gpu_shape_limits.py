"""Molecules near the kernels' shared-memory limit, where the launch plans go without the
factors, or the AO slots, in shared memory (at one walker per block nothing else fits): psi,
local energies, Metropolis chains, position gradients, adjoints and both gradient samplers
against the oracle, or against the same molecule's other kernels."""
import numpy as np
import pytest
import torch

from oracle import qmc_oracle as orc
from tests.test_gpu_s_contractions import molecule

pytestmark = pytest.mark.gpu

WEIGHT = 50.0  # of the Jastrow factor: with less, exp(log J) of so many pairs overflows


def system(natom, nfun, nw=5):
    mol = molecule(nfun, natom, 3.0)
    order = np.concatenate([np.arange(0, natom, 2), np.arange(1, natom, 2)])  # a spin per atom
    centers = np.asarray(mol.atom_coords)[order]
    pos = centers[None] + 0.7 * np.random.default_rng(natom).normal(size=(nw, natom, 3))
    return mol, pos.reshape(nw, -1)


def wave(mol, **kw):
    from qmctorch_gb300.wavefunction import SlaterJastrow
    torch.set_default_dtype(torch.float64)
    wf = SlaterJastrow(mol, cuda=True, include_all_mo=False, **kw)
    wf.jastrow.jastrow_kernel.weight.data.fill_(WEIGHT)
    return wf


# atoms, functions per atom: factors in the work arrays (FP64 local energy); sums of FP64
# multiply-adds (FP64 local energy; psi)
@pytest.mark.parametrize("natom,nfun,eloc", [(108, 1, True), (72, 6, True), (80, 6, False)])
def test_fp64(natom, nfun, eloc):
    from qmctorch_gb300.sampler import Metropolis
    mol, pos = system(natom, nfun)
    wf, x = wave(mol), torch.as_tensor(pos, device="cuda")
    ow = orc.OracleSlaterJastrow(mol, include_all_mo=False, jastrow_w=WEIGHT)
    with torch.no_grad():
        np.testing.assert_allclose(wf(x).cpu().numpy(), ow.forward(pos), rtol=1e-9)
        if eloc:
            np.testing.assert_allclose(wf.local_energy(x).cpu().numpy(), ow.local_energy(pos),
                                       rtol=1e-8)
    out = []
    for nw in (5, 1):  # each walker's chain does not depend on the others
        s = Metropolis(nwalkers=nw, nstep=4, step_size=0.05, ntherm=-1, nelec=natom, ndim=3,
                       init=mol.domain("atomic"), cuda=True, seed=3,
                       move={"type": "all-elec", "proba": "normal"})
        out.append(s(wf.pdf, pos=x[:nw].clone(), with_tqdm=False).detach().cuda())
    assert torch.equal(out[0][:1], out[1]) and not torch.equal(out[0], x)


# factors in the work arrays; columns in registers, a pass per eight
@pytest.mark.parametrize("natom,nfun", [(120, 2), (96, 6)])
def test_mixed_local_energy(natom, nfun):
    mol, pos = system(natom, nfun)
    ow = orc.OracleSlaterJastrow(mol, include_all_mo=False, jastrow_w=WEIGHT)
    with torch.no_grad():
        got = wave(mol, precision="mixed").local_energy(torch.as_tensor(pos, device="cuda"))
    np.testing.assert_allclose(got.cpu().numpy(), ow.local_energy(pos), rtol=2e-3)

