"""Metropolis decisions where psi^2 is below FP64's normal range (far-off walkers of larger
molecules): orbitals scaled by a power of two leave every ratio of densities as it is, so the
chain has to be that of the unscaled orbitals, as long as no density is zero."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bits", [0, 100, 255])
@pytest.mark.parametrize("move", ["all-elec", "all-elec-iter"])
def test_scaled_orbitals_give_the_same_chain(move, bits):
    from qmctorch_gb300.sampler import Metropolis
    from qmctorch_gb300.scf import Molecule
    from qmctorch_gb300.wavefunction import SlaterJastrow
    torch.set_default_dtype(torch.float64)
    mol = Molecule("H 0 0 -0.37; H 0 0 0.37", unit="angs", basis="sto-3g", calculator="huckel")
    g = torch.Generator().manual_seed(4)
    x = torch.as_tensor(mol.atom_coords).reshape(1, 6) + 0.3 * torch.randn((300, 6), generator=g)
    out = []
    for scale in (1.0, 2.0 ** -bits):
        # two configurations: the all-electron kernel also for single-electron moves
        wf = SlaterJastrow(mol, configs="single_double(2,2)", cuda=True)
        wf.fc.weight.data[0, 1:] = 0.125
        wf.mo.mo_modifier.data *= scale
        s = Metropolis(nwalkers=300, nstep=20, step_size=0.3, ntherm=-1, nelec=2, ndim=3,
                       init=mol.domain("atomic"), cuda=True, seed=5,
                       move={"type": move, "proba": "normal"})
        out.append(s(wf.pdf, pos=x.clone().cuda(), with_tqdm=False))
        if scale == 1.0:
            # psi^2 within 2^-24 .. 1: at 2^-1020 of it 2^-1044 and more, 30 bits above the
            # smallest number, so a decision differs by rounding with a chance of 2^-29 per move
            assert float(wf.pdf(out[0]).detach().min()) > 2.0 ** -24 and float(wf.pdf(x.cuda()).detach().min()) > 2.0 ** -24
        elif bits == 255:
            assert 0 < float(wf(x.cuda()).detach().abs().max()) < 2.0 ** -505
    assert not torch.equal(out[0], x.cuda())
    assert torch.equal(out[0], out[1])
