"""Orbitals next to their nodal plane, where the AOs that an orbital has are small against
the others of the electron: the AO -> MO layer's entries, and psi, E_L, gradients and adjoints
of molecules with one electron per spin (whose determinants are such entries), keep their own
relative accuracy."""
import numpy as np
import pytest
import torch

from oracle import qmc_oracle as orc

pytestmark = pytest.mark.gpu


def water(cuda=True):
    from qmctorch_gb300.scf import Molecule
    from qmctorch_gb300.wavefunction import SlaterJastrow
    torch.set_default_dtype(torch.float64)
    mol = Molecule("O 0 0 0.1173; H 0 0.7572 -0.4692; H 0 -0.7572 -0.4692", unit="angs",
                   basis="cc-pvdz", calculator="huckel")
    return mol, SlaterJastrow(mol, cuda=cuda)


@pytest.mark.parametrize("z", [1.0, 1e-3, 1e-6, 1e-9])
def test_layer_entries(z):
    mol, wf = water()
    wf.mo.mo_scf[wf.mo.mo_scf.abs() < 1e-9] = 0.0
    x = torch.as_tensor(np.random.default_rng(1).normal(size=(300, 10, 3)), device="cuda")
    x[:, :, 0] *= z  # the molecule's plane is x = 0
    with torch.no_grad():
        ao = wf.ao(x.reshape(300, 30))
        mo, w = wf.mo(ao), wf.mo.mo_scf * wf.mo.mo_modifier
    # 25 AOs in two chunks of limbs: at most 50 x 2^-60 of the largest product that they could
    # have, of which an entry is 2^-12 at least, else it is formed by multiply-adds
    assert ((mo - ao @ w).abs() <= 2.0 ** -42 * (ao.abs() @ w.abs())).all()


def test_layer_entries_in_many_columns():
    """80 orbitals in slices of 72 and 8 columns, AOs of all magnitudes; infinities and NaN."""
    from tests.test_gpu_s_contractions import molecule
    from qmctorch_gb300.wavefunction import SlaterJastrow
    mol, rng = molecule(2, 40), np.random.default_rng(4)
    mol.basis.mos, mol.basis.nmo = rng.normal(size=(80, 80)), 80
    wf = SlaterJastrow(mol, cuda=True)
    ao = torch.as_tensor(rng.normal(size=(333, 80)) * 10.0 ** rng.uniform(-12, 1, size=(333, 80)))
    ao[7], ao[8, 3], ao[9, 5] = 0.0, np.inf, np.nan
    ao = ao.cuda()
    with torch.no_grad():
        mo, w = wf.mo(ao), wf.mo.mo_scf * wf.mo.mo_modifier
    want = ao @ w
    rows = torch.ones(333, dtype=torch.bool)
    rows[8:10] = False
    # 80 AOs in six chunks: 160 x 2^-60 of the largest product, an entry at least 2^-12 of it
    assert ((mo - want).abs() <= 2.0 ** -40 * (ao.abs() @ w.abs()))[rows].all()
    assert torch.equal(mo[8], want[8]) and torch.isnan(mo[9]).all()


@pytest.mark.parametrize("z", [1.0, 1e-3, 1e-6, 1e-9])
def test_one_electron_per_spin(z):
    """H2 with its electrons in an orbital of p functions along x (and in a second one)."""
    from qmctorch_gb300.scf import Molecule
    from qmctorch_gb300.wavefunction import SlaterJastrow
    torch.set_default_dtype(torch.float64)
    mol = Molecule("H 0 0 -0.37; H 0 0 0.37", unit="angs", basis="cc-pvdz", calculator="huckel")
    b = mol.basis
    px = np.zeros(b.nao)
    px[np.asarray(b.index_ctr)[np.asarray(b.bas_kx) == 1]] = 1.0
    mos = np.asarray(b.mos).copy()
    mos[:, 0], mos[:, 1] = 0.7 * px, 0.4 * px * np.where(np.arange(b.nao) < b.nao // 2, 1, -1)
    b.mos = mos
    wf = SlaterJastrow(mol, configs="single_double(2,2)", cuda=True)
    c = np.random.default_rng(3).uniform(0.3, 1.0, size=wf.nci)
    wf.fc.weight.data = torch.as_tensor(c, device="cuda").reshape(1, -1)
    pos = np.random.default_rng(2).normal(size=(200, 2, 3))
    pos[:, :, 0] *= z
    pos = pos.reshape(200, 6)
    x = torch.as_tensor(pos, device="cuda")
    ow = orc.OracleSlaterJastrow(mol, configs="single_double(2,2)", fc_weight=c)
    psi, el = ow.forward(pos).reshape(-1), ow.local_energy(pos).reshape(-1)
    # relative errors of some units of 2^-52, amplified where the configurations cancel
    scale = np.abs(orc.OracleSlaterJastrow(mol, configs="single_double(2,2)",
                                           fc_weight=np.eye(wf.nci)[0]).forward(pos)).reshape(-1)
    with torch.no_grad():
        got, gel = wf(x).cpu().numpy().reshape(-1), wf.local_energy(x).cpu().numpy().reshape(-1)
    assert (np.abs(got - psi) <= 1e-13 * np.maximum(scale, np.abs(psi))).all()
    keep = np.abs(psi) > 1e-2 * scale
    assert keep.sum() > 100
    np.testing.assert_allclose(gel[keep], el[keep], rtol=1e-10, atol=1e-10)
    # psi is proportional to x of each electron close to the plane: d log psi / dx = 1 / x
    g = (wf.gradients(x).cpu().numpy() / psi[:, None])[:, ::3]
    if z <= 1e-6:
        np.testing.assert_allclose((g * pos[:, ::3])[keep], 1.0, rtol=1e-9)
    gel = wf._adjoint(x[torch.as_tensor(keep)], torch.ones(int(keep.sum())).cuda(),
                      "qmc_wf_local_energy_adjoint", "qmc_eloc_adjoint_scratch_bytes")
    # E_L does not change when all configurations grow alike, nor when both orbitals do
    total = float((gel[4].reshape(-1).cpu() * torch.as_tensor(c)).sum())
    assert abs(total) <= 1e-9 * float((gel[4].reshape(-1).cpu().abs() * torch.as_tensor(c)).sum())
