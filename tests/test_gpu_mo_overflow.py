"""Orbital coefficients so large that MO values leave FP64's range: psi is not finite, as with
multiply-adds."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def water(**kw):
    from qmctorch_gb300.scf import Molecule
    from qmctorch_gb300.wavefunction import SlaterJastrow
    torch.set_default_dtype(torch.float64)
    mol = Molecule("O 0 0 0.1173; H 0 0.7572 -0.4692; H 0 -0.7572 -0.4692", unit="angs",
                   basis="cc-pvdz", calculator="huckel")
    wf = SlaterJastrow(mol, configs="single_double(4,4)", cuda=True, **kw)
    wf.fc.weight.data = torch.as_tensor(np.random.default_rng(5).uniform(size=(1, wf.nci))).cuda()
    return mol, wf


def test_mo_values_beyond_the_range_are_infinite():
    from qmctorch_gb300.serving import seeded_positions
    mol, wf = water()
    x = torch.as_tensor(seeded_positions(mol, 100, 4), device="cuda")
    x[:50, :3] = torch.as_tensor(np.asarray(mol.atom_coords)[0] + 0.01)  # at the oxygen nucleus
    with torch.no_grad():
        mo = (wf.ao(x) @ wf.mo.mo_scf)[..., 0].abs()
        assert torch.isfinite(wf(x)).all()
        wf.mo.mo_modifier.data[:, 0] = 2.0 ** 1022
        over = (mo > 4).any(1)  # |MO| 2^1022 > 2^1024 for an electron of the walker
        assert over[:50].all()
        assert not torch.isfinite(wf(x)[over]).any()
