"""Exponent gradients of primitives whose exponential is far below 1e-20 at every electron:
the adjoint sums them all the same, as the derivative's definition does."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def test_exponent_gradients_of_far_primitives():
    from qmctorch_gb300.scf import Molecule
    from qmctorch_gb300.wavefunction import SlaterJastrow
    torch.set_default_dtype(torch.float64)
    mol = Molecule("H 0 0 -0.37; H 0 0 0.37", unit="angs", basis="sto-3g", calculator="huckel")
    wf = SlaterJastrow(mol, cuda=True)
    # alpha r^2 of 50 to 90 for the middle primitives (0.62) and of 280 to 490 for the tightest
    # (3.4), both cut in the forward pass; the widest (0.17) stay below 46
    r = np.linspace(9.0, 12.0, 20)
    pos = np.zeros((20, 2, 3))
    pos[:, 0, 0], pos[:, 1, 1] = r, -r
    x = torch.as_tensor(pos.reshape(20, 6), device="cuda")
    b = mol.basis
    alpha = torch.as_tensor(np.asarray(b.bas_exp)).requires_grad_(True)
    weight = torch.as_tensor((2 * np.asarray(b.bas_exp) / np.pi) ** 0.75 * np.asarray(b.bas_coeffs))
    atom = torch.as_tensor(np.asarray(mol.atom_coords))[np.repeat([0, 1], 3)]
    d = torch.as_tensor(pos).unsqueeze(2) - atom
    ao = (weight * torch.exp(-alpha * (d * d).sum(-1))).reshape(20, 2, 2, 3).sum(-1)
    phi = ao @ wf.mo.mo_scf.cpu()[:, 0]
    u = 0.5 * (q := torch.as_tensor(pos[:, 0] - pos[:, 1]).norm(dim=-1)) / (1 + q)
    psi = torch.exp(u) * phi[:, 0] * phi[:, 1]
    for i in range(20):
        want, = torch.autograd.grad(psi[i], alpha, retain_graph=True)
        for p in wf.parameters():
            p.grad = None
        wf(x[i:i + 1]).sum().backward()
        got = wf.ao.bas_exp.grad.cpu()
        np.testing.assert_allclose(got.numpy(), want.numpy(), rtol=1e-10)
