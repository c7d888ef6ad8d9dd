"""The fused kernels sum the radial part of a p or d shell once when its components share
their weights, component by component otherwise: both against psi and E_L pieces from the
layers, which evaluate every AO by itself."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scaled", [(), (0,), (1,), (2, 5), (-1,)])
@pytest.mark.parametrize("precision,rtol", [("fp64", 1e-10), ("mixed", 1e-3)])
def test_weights_that_differ_between_components(scaled, precision, rtol):
    from qmctorch_gb300.scf import Molecule
    from qmctorch_gb300.serving import seeded_positions
    from qmctorch_gb300.wavefunction import SlaterJastrow
    torch.set_default_dtype(torch.float64)
    mol = Molecule("O 0 0 0.1173; H 0 0.7572 -0.4692; H 0 -0.7572 -0.4692", unit="angs",
                   basis="cc-pvdz", calculator="huckel")
    wf = SlaterJastrow(mol, configs="single_double(4,4)", cuda=True, precision=precision)
    wf.fc.weight.data = torch.as_tensor(np.random.default_rng(5).uniform(size=(1, wf.nci))).cuda()
    # the components of the oxygen d shell (one primitive each) and of its first p shell
    tables = wf.ao.device_tables(torch.device("cuda", torch.cuda.current_device())).t
    k = np.asarray(mol.basis.bas_kx) + np.asarray(mol.basis.bas_ky) + np.asarray(mol.basis.bas_kz)
    entry = tables["w_entry"].cpu().numpy()
    for shell in (2, 1):
        first = int(np.flatnonzero(k[entry] == shell)[0])
        for c in scaled:
            tables["ao_wd"][first + (c if shell == 2 else 0)] *= 1.0 + 0.125 * (1 + abs(c))
    x = torch.as_tensor(seeded_positions(mol, 300, 4), device="cuda")
    with torch.no_grad():
        wf.mo.precision = "fp64"
        want = wf(x, ao=wf.ao(x)).cpu().numpy()
        got = wf(x).cpu().numpy()
    np.testing.assert_allclose(got, want, rtol=rtol, atol=rtol * np.abs(want).max() * 1e-3)
