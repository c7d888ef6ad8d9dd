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


# the instances with eight columns, without limbs, and with the adjoints' tile in the scratch
@pytest.mark.parametrize("natom,nfun", [(80, 6), (100, 4), (94, 5), (120, 3)])
def test_gradient_kernels(natom, nfun):
    from qmctorch_gb300.sampler import GeneralizedMetropolis, Hamiltonian
    mol, pos = system(natom, nfun, nw=3)
    wf, x, rng = wave(mol), torch.as_tensor(pos, device="cuda"), np.random.default_rng(1)
    exps, shape = np.asarray(mol.basis.bas_exp), (mol.basis.nao, natom // 2)
    de, dm, dx = rng.normal(size=exps.shape) * exps, rng.normal(size=shape), rng.normal(size=pos.shape)
    h = 1e-6

    def log_psi(t=0.0, tx=0.0, eloc=False):
        ow = orc.OracleSlaterJastrow(mol, include_all_mo=False, jastrow_w=WEIGHT + t,
                                     mo_modifier=1 + t * dm, bas_exp=exps + t * de)
        p = pos + tx * dx
        return (ow.local_energy(p) if eloc else np.log(np.abs(ow.forward(p)))).reshape(-1)

    psi = torch.as_tensor(orc.OracleSlaterJastrow(mol, include_all_mo=False, jastrow_w=WEIGHT)
                          .forward(pos).reshape(-1), device="cuda")
    # central differences: an error of h^2 beside rounding (1e-13) over h
    grad = (wf.gradients(x) / psi[:, None]).cpu().numpy()
    want = (log_psi(tx=h) - log_psi(tx=-h)) / (2 * h)
    np.testing.assert_allclose((grad * dx).sum(1), want, rtol=1e-5, atol=1e-5 * np.abs(want).max())
    for kind, eloc in (("", False), ("_local_energy", True)):
        fn = "qmc_wf%s_adjoint" % (kind or "_psi")
        gout = torch.ones_like(psi) if eloc else 1 / psi
        g = wf._adjoint(x, gout, fn, "qmc_eloc_adjoint_scratch_bytes" if eloc
                        else "qmc_adjoint_scratch_bytes")
        got = [float((g[0].cpu() * torch.as_tensor(de)).sum()),
               float((g[1].cpu()[:, :natom // 2] * torch.as_tensor(dm)).sum()), float(g[2].sum())]
        want = ((log_psi(h, eloc=eloc) - log_psi(-h, eloc=eloc)) / (2 * h)).sum()
        assert abs(sum(got) - want) <= 2e-5 * max(map(abs, got)), (got, want)
    common = dict(nwalkers=3, ntherm=-1, nelec=natom, ndim=3, cuda=True, seed=2)
    # a leapfrog trajectory whose force is the gradient of log psi^2 keeps its energy
    out = Hamiltonian(nstep=1, step_size=1e-3, L=2, **common)(wf.pdf, pos=x.clone(), with_tqdm=False)
    assert torch.isfinite(out).all() and (out.cuda() != x).any(1).all()
    cfg = tuple(torch.arange(natom // 2).reshape(1, -1) for _ in range(2))
    outs = []
    for w in (wf, wave(mol, configs=cfg)):
        s = GeneralizedMetropolis(nstep=3, step_size=0.05, **common)
        outs.append(s(w.pdf, pos=x.clone(), with_tqdm=False).detach())
    assert torch.isfinite(outs[0]).all() and (outs[0] - outs[1]).abs().max() < 1e-8
