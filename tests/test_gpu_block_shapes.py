"""Shapes at which blocks, tiles and column groups are partly empty: the layers' kernels
against dense products of their own inputs, the fused psi against the layers, the sweep
kernel's walkers against the same walkers in another grid."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

MOLECULES = {"H2": ("H 0 0 -0.37; H 0 0 0.37", "sto-3g"),
             "LiH": ("Li 0 0 0; H 0 0 1.595", "sto-3g"),
             "H2O": ("O 0 0 0.1173; H 0 0.7572 -0.4692; H 0 -0.7572 -0.4692", "cc-pvdz"),
             "H18": ("; ".join("H 0 0 %g" % (0.95 * i) for i in range(18)), "sto-3g")}


def wave(name, **kw):
    from qmctorch_gb300.scf import Molecule
    from qmctorch_gb300.wavefunction import SlaterJastrow
    torch.set_default_dtype(torch.float64)
    atoms, basis = MOLECULES[name]
    mol = Molecule(atoms, unit="angs", basis=basis, calculator="huckel")
    return mol, SlaterJastrow(mol, cuda=True, **kw)


@pytest.mark.parametrize("nw", [1, 31, 130])
@pytest.mark.parametrize("all_mo", [False, True])
@pytest.mark.parametrize("name", sorted(MOLECULES))
def test_layers(name, all_mo, nw):
    from qmctorch_gb300.serving import seeded_positions
    mol, wf = wave(name, include_all_mo=all_mo)
    x = torch.as_tensor(seeded_positions(mol, nw, 2), device="cuda")
    with torch.no_grad():
        ao = wf.ao(x)
        mo = wf.mo(ao)
        w = wf.mo.mo_scf * wf.mo.mo_modifier
        want, scale = ao @ w, ao.abs() @ w.abs()
        # fixed point relative to the largest products: 2^-50 of them per chunk of AOs
        assert ((mo - want).abs() <= 1e-13 * scale.amax(-1, keepdim=True)).all()
        psi = wf(x)
        assert ((wf(x, ao=ao) - psi).abs() <= 1e-9 * psi.abs().clamp_min(1e-3 * psi.abs().max())).all()


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_sweep_grids(precision):
    from qmctorch_gb300.sampler import Metropolis
    from qmctorch_gb300.serving import seeded_positions
    mol, wf = wave("H18", precision=precision)
    x = torch.as_tensor(seeded_positions(mol, 152 * 24 + 1, 2), device="cuda")
    out = {}
    for nw in (1, 23, 25, 152 * 16 + 1, 152 * 24 + 1):
        s = Metropolis(nwalkers=nw, nstep=2, step_size=0.1, ntherm=-1, nelec=mol.nelec, ndim=3,
                       init=mol.domain("atomic"), cuda=True, seed=5,
                       move={"type": "all-elec-iter", "proba": "normal"})
        out[nw] = s(wf.pdf, pos=x[:nw].clone(), with_tqdm=False)
        assert not torch.equal(out[nw], x[:nw])
    last = out[152 * 24 + 1]
    for nw, o in out.items():
        assert torch.equal(o, last[:nw])
