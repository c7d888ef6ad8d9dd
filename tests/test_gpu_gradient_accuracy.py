"""Position gradients and the adjoints' parameter gradients where a spin's excitation ratios
are large but not extreme: as accurate as the same configurations given as an explicit list.
More than sixteen orbital columns: excitation mode against an explicit list."""
import numpy as np
import pytest
import torch

from tests.test_gpu_large_ratio import columns

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def waves():
    """Excitation-mode and explicit-mode H2O, walkers with ratios of 100 to 4000."""
    from qmctorch_gb300.scf import Molecule
    from qmctorch_gb300.serving import seeded_positions
    from qmctorch_gb300.wavefunction import SlaterJastrow
    torch.set_default_dtype(torch.float64)
    mol = Molecule("O 0 0 0.1173; H 0 0.7572 -0.4692; H 0 -0.7572 -0.4692", unit="angs",
                   basis="cc-pvdz", calculator="huckel")
    wf = SlaterJastrow(mol, configs="single_double(4,4)", cuda=True)
    tab = wf.pool._tables
    cfg = tuple(columns(tab, s, 5)[tab.t["cfg_det%d" % s].cpu().long()] for s in range(2))
    ex = SlaterJastrow(mol, configs=cfg, cuda=True)
    weight = torch.as_tensor(np.random.default_rng(5).uniform(0.2, 1.0, size=(1, wf.nci))).cuda()
    for w in (wf, ex):
        w.fc.weight.data = weight.clone()
    x = torch.as_tensor(seeded_positions(mol, 40_000, 9), device="cuda")
    with torch.no_grad():
        mo, ratio = wf.mo(wf.ao(x)), 0
        for s in range(2):
            m = mo[:, 5 * s:5 * s + 5]
            d = torch.stack([torch.linalg.det(m[:, :, c]) for c in columns(tab, s, 5).cuda()], 1)
            ratio = torch.maximum(d.abs().amax(1) / d[:, 0].abs(), torch.as_tensor(ratio).cuda())
    keep = (ratio > 100) & (ratio < 4000)
    assert int(keep.sum()) > 200
    return wf, ex, x[keep][:1000].contiguous()


def test_position_gradients(waves):
    wf, ex, x = waves
    got, want = wf.gradients(x), ex.gradients(x)
    # rounding of both, amplified by matrices of condition 1e3; a formula that loses the
    # ratio's square has 1e-12 and more
    assert ((got - want).abs().amax(1) <= 2e-13 * want.abs().amax(1)).all()


@pytest.mark.parametrize("kind", ["psi", "eloc"])
def test_parameter_gradients(waves, kind):
    wf, ex, x = waves
    for chunk in x.split(50):  # few walkers: no cancellation between them
        grads = []
        for w in (wf, ex):
            for p in w.parameters():
                p.grad = None
            (w(chunk) if kind == "psi" else w.local_energy(chunk)).sum().backward()
            grads.append([w.ao.bas_exp.grad, w.mo.mo_modifier.grad, w.fc.weight.grad])
        for got, want in zip(*grads):
            assert (got - want).norm() <= 1e-12 * want.norm()


@pytest.mark.parametrize("nw", [3, 40])
def test_more_than_sixteen_columns(nw):
    """C6H6, 21 orbitals: gradients, adjoints, drift and HMC of the ground-state determinant."""
    from qmctorch_gb300.sampler import GeneralizedMetropolis, Hamiltonian
    from qmctorch_gb300.scf import Molecule
    from qmctorch_gb300.serving import seeded_positions
    from qmctorch_gb300.wavefunction import SlaterJastrow
    torch.set_default_dtype(torch.float64)
    ring = [(np.cos(np.pi * i / 3), np.sin(np.pi * i / 3)) for i in range(6)]
    atoms = "; ".join("%s %.6f %.6f 0" % (a, r * c, r * s) for a, r in (("C", 1.39), ("H", 2.48))
                      for c, s in ring)
    mol = Molecule(atoms, unit="angs", basis="sto-3g", calculator="huckel")
    cfg = tuple(torch.arange(21).reshape(1, -1) for _ in range(2))
    pair = [SlaterJastrow(mol, cuda=True), SlaterJastrow(mol, configs=cfg, cuda=True)]
    x = torch.as_tensor(seeded_positions(mol, nw, 4), device="cuda")
    got, want = (w.gradients(x) for w in pair)
    assert ((got - want).abs() <= 1e-9 * want.abs().amax(1, keepdim=True)).all()
    for kind in ("psi", "eloc"):
        grads = []
        for w in pair:
            for p in w.parameters():
                p.grad = None
            psi = w(x)
            ((psi / psi.detach()) if kind == "psi" else w.local_energy(x)).sum().backward()
            grads.append([w.ao.bas_exp.grad, w.mo.mo_modifier.grad,
                          w.jastrow.jastrow_kernel.weight.grad])
        for a, b in zip(*grads):
            assert (a - b).norm() <= 1e-8 * b.norm()
    common = dict(nwalkers=nw, ntherm=-1, nelec=42, ndim=3, cuda=True, rng="torch")
    for make in (lambda: GeneralizedMetropolis(nstep=6, step_size=0.05, **common),
                 lambda: Hamiltonian(nstep=1, step_size=0.01, L=3, **common)):
        out = []
        for w in pair:
            torch.manual_seed(3)
            out.append(make()(w.pdf, pos=x.clone(), with_tqdm=False).detach().cuda())
        assert (out[1] != x).any()
        assert (out[0] - out[1]).abs().max() < 1e-8
