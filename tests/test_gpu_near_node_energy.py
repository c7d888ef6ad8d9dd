"""Local energies next to a node of the ground determinant, where excitation ratios of K
amplify the rounding of A^-1 by K^2 in the excitation formulas: as accurate as the same
configurations given as an explicit list, whose kernel factors every determinant."""
import numpy as np
import pytest
import torch

from tests.test_gpu_large_ratio import columns, waves  # noqa: F401 (a fixture)

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nw", [1, 17, 64])
def test_energies_are_those_of_the_explicit_list(waves, nw):  # noqa: F811
    wf, ex, x, ratio = waves
    with torch.no_grad():
        got, want = wf.local_energy(x[:nw]).reshape(-1), ex.local_energy(x[:nw]).reshape(-1)
    # ratios of 5e3 to 2e5 leave 1e-9 to 1e-6 in the excitation formulas; the determinants
    # themselves have matrices of condition 1e3 to 1e4
    assert ((got - want).abs() <= 1e-11 * (1 + want.abs())).all()


def test_one_electron_in_its_nodal_plane(waves):  # noqa: F811
    """det A is zero and excited determinants are not: the energy is finite and that of the
    explicit list."""
    from qmctorch_gb300.wavefunction import SlaterJastrow
    wf, _, x, _ = waves
    tab = wf.pool._tables
    cfg = tuple(columns(tab, s, 5)[tab.t["cfg_det%d" % s].cpu().long()] for s in range(2))
    out = []
    y = torch.as_tensor(np.random.default_rng(2).normal(size=(64, 10, 3))).cuda() * 0.7
    y = y + torch.as_tensor(np.asarray(wf.mol.atom_coords))[0].cuda()
    y[:, :5, 0] = 0.0
    y = y.reshape(64, 30)
    for configs in ("single_double(4,4)", cfg):
        w = SlaterJastrow(wf.mol, configs=configs, cuda=True)
        w.mo.mo_scf[w.mo.mo_scf.abs() < 1e-9] = 0.0
        w.fc.weight.data = wf.fc.weight.data.clone()
        with torch.no_grad():
            out.append(w.local_energy(y).reshape(-1))
    keep = out[1].abs() < 1e3  # not at a node of psi itself
    assert int(keep.sum()) > 8
    assert ((out[0] - out[1]).abs()[keep] <= 1e-10 * (1 + out[1].abs()[keep])).all()
