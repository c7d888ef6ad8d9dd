"""Groups of one to six s functions over one exponent set (general contractions): the AO
layer and the fused kernels against the oracle. A group's last functions are the last of an
electron's row, where a kernel that takes the group for a larger one writes past it."""
import types

import numpy as np
import pytest
import torch

from oracle import qmc_oracle as orc

pytestmark = pytest.mark.gpu


def molecule(nfun, natom=6, spacing=0.95):
    """A chain of hydrogen atoms in sto-3g, ``nfun`` contractions of each one's primitives."""
    from qmctorch_gb300.scf import Molecule
    torch.set_default_dtype(torch.float64)
    mol = Molecule("; ".join("H 0 0 %g" % (spacing * i) for i in range(natom)), unit="angs",
                   basis="sto-3g", calculator="huckel")
    b, rng = mol.basis, np.random.default_rng(nfun)
    at = np.asarray(b.index_ctr).reshape(natom, 3)  # entries of an atom: three primitives
    take = np.repeat(np.arange(natom), nfun)    # the atom of each new function
    entry = np.concatenate([np.flatnonzero(np.isin(b.index_ctr, at[a])) for a in take])
    new = types.SimpleNamespace(**vars(b))
    for key in ("bas_exp", "bas_n", "bas_l", "bas_kr", "bas_kx", "bas_ky", "bas_kz", "bas_norm"):
        setattr(new, key, np.asarray(getattr(b, key))[entry])
    scale = np.where(np.arange(natom * nfun) % nfun == 0, 1.0, 0.0)[:, None]
    new.bas_coeffs = (np.asarray(b.bas_coeffs)[entry].reshape(-1, 3) * scale
                      + (1 - scale) * rng.uniform(0.1, 0.6, size=(natom * nfun, 3))).reshape(-1)
    new.index_ctr = np.repeat(np.arange(natom * nfun), 3)
    new.nshells = np.full(natom, 3 * nfun)
    new.nao_per_atom = np.full(natom, nfun)
    new.nctr_per_ao = np.full(natom * nfun, 3)
    new.nao = natom * nfun
    new.mos = scale * np.asarray(b.mos)[take] + (1 - scale) * rng.normal(
        scale=0.1, size=(natom * nfun, np.asarray(b.mos).shape[1]))
    mol.basis = new
    return mol


@pytest.mark.parametrize("nfun", [1, 2, 3, 4, 5, 6])
def test_s_contractions(nfun):
    from qmctorch_gb300.serving import seeded_positions
    from qmctorch_gb300.wavefunction import SlaterJastrow
    mol = molecule(nfun)
    wf = SlaterJastrow(mol, cuda=True)
    assert wf.ao._tables.groups == [(nfun * a, nfun * a + nfun) for a in range(6)]
    ow = orc.OracleSlaterJastrow(mol)
    pos = seeded_positions(mol, 70, 3)
    x = torch.as_tensor(pos, device="cuda")
    r = pos.reshape(-1, 1, 3) - np.asarray(mol.atom_coords)[np.repeat(np.arange(6), nfun)]
    b = mol.basis
    norm = ((2 * b.bas_exp / np.pi) ** 0.75 * b.bas_coeffs).reshape(-1, 3)
    a, r2 = b.bas_exp.reshape(-1, 3), (r ** 2).sum(-1)[..., None]
    e = norm * np.exp(-a * r2)
    want = (e.sum(-1), -2 * (a * e).sum(-1)[..., None] * r, ((4 * a * a * r2 - 6 * a) * e).sum(-1))
    with torch.no_grad():
        for got, w in zip(wf.ao(x, derivative=[0, 1, 2], sum_grad=False, sum_hess=True), want):
            got = got.cpu().numpy().reshape(w.shape)
            np.testing.assert_allclose(got, w, rtol=1e-11, atol=1e-12)
        np.testing.assert_allclose(wf.ao(x).cpu().numpy().reshape(want[0].shape), want[0],
                                   rtol=1e-11, atol=1e-12)
        psi = ow.forward(pos).reshape(-1)
        np.testing.assert_allclose(wf(x).cpu().numpy().reshape(-1), psi, rtol=1e-9,
                                   atol=1e-12 * np.abs(psi).max())
        # E_L amplifies rounding by the condition of the Slater matrices (some 1e3)
        np.testing.assert_allclose(wf.local_energy(x).cpu().numpy().reshape(-1),
                                   ow.local_energy(pos).reshape(-1), rtol=1e-8)
        mixed = SlaterJastrow(mol, cuda=True, precision="mixed")(x).cpu().numpy().reshape(-1)
        np.testing.assert_allclose(mixed, psi, rtol=1e-3, atol=1e-4 * np.abs(psi).max())
