"""The drift and HMC samplers from walkers next to, and exactly at, a node of the ground
determinant where excited ones do not vanish, against the same configurations as an explicit
list (whose kernels factor every determinant): moves that are accepted and rejected, with the
drift and the force of each in the positions that are compared."""
import numpy as np
import pytest
import torch

from tests.test_gpu_large_ratio import columns, waves  # noqa: F401 (a fixture)

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def starts(waves):  # noqa: F811
    """name -> (excitation-mode wave function, explicit one, walkers): ratios of 5e3 to 2e5;
    the up electrons, or all, in the nodal plane of the highest occupied orbital, whose
    coefficients of other symmetries are exactly zero: det A = 0."""
    wf, ex, x, _ = waves
    out = {"near": (wf, ex, x)}
    for spins in ("up", "both"):
        from qmctorch_gb300.wavefunction import SlaterJastrow
        pair = []
        for w in (wf, ex):
            cfg = "single_double(4,4)" if w is wf else ex_configs(wf)
            v = SlaterJastrow(w.mol, configs=cfg, cuda=True)
            v.mo.mo_scf[v.mo.mo_scf.abs() < 1e-9] = 0.0
            v.fc.weight.data = w.fc.weight.data.clone()
            pair.append(v)
        y = torch.as_tensor(np.random.default_rng(2).normal(size=(64, 10, 3))).cuda()
        y = y * 0.7 + torch.as_tensor(np.asarray(wf.mol.atom_coords))[0].cuda()
        y[:, : 5 if spins == "up" else 10, 0] = 0.0
        y = y.reshape(64, 30)
        mo = pair[0].mo(pair[0].ao(y)).detach()
        det = torch.linalg.det(mo[:, :5, :5])
        assert (det == 0).all() and (pair[1](y).abs() > 0).any()
        # walkers at a node of psi itself have no drift: keep those with a moderate one
        drift = pair[1].gradients(y) / pair[1](y).detach().reshape(-1, 1)
        out[spins] = pair[0], pair[1], y[(drift.abs().amax(1) < 30)][:32].contiguous()
        assert len(out[spins][2]) > 8
    return out


def ex_configs(wf):
    tab = wf.pool._tables
    return tuple(columns(tab, s, 5)[tab.t["cfg_det%d" % s].cpu().long()] for s in range(2))


@pytest.mark.parametrize("name", ["near", "up", "both"])
def test_drift(starts, name):
    from qmctorch_gb300.sampler import GeneralizedMetropolis
    wf, ex, x = starts[name]
    out = []
    for w in (wf, ex):
        torch.manual_seed(3)
        s = GeneralizedMetropolis(nwalkers=len(x), nstep=8, step_size=0.05, ntherm=0, ndecor=1,
                                  nelec=10, ndim=3, cuda=True, rng="torch")
        out.append(s(w.pdf, pos=x.clone(), with_tqdm=False).detach().reshape(-1, len(x), 30))
    steps = torch.cat([x[None], out[1]])
    moved = (steps[1:] != steps[:-1]).any(-1)
    assert moved.any() and (~moved).any()
    # the drift, at most some 1e4, times the step and FP64 rounding amplified by the
    # condition of the matrices (1e4)
    assert (out[0] - out[1]).abs().max() < 1e-8


@pytest.mark.parametrize("name", ["near", "up", "both"])
def test_hmc(starts, name):
    from qmctorch_gb300.sampler import Hamiltonian
    wf, ex, x = starts[name]
    drift = ex.gradients(x) / ex(x).detach().reshape(-1, 1)
    x = x[drift.abs().amax(1) < 30].contiguous()  # not at a node of psi: no steep force
    assert len(x) > 4
    out = []
    for w in (wf, ex):
        torch.manual_seed(3)
        s = Hamiltonian(nwalkers=len(x), nstep=1, step_size=0.01, L=3, ntherm=0, nelec=10, ndim=3,
                        cuda=True, rng="torch")
        out.append(s(w.pdf, pos=x.clone(), with_tqdm=False).detach().reshape(len(x), 30))
    moved = (out[1] != x).any(-1)
    assert moved.any()
    # the force (2 grad log psi, some 10) enters with the square of the time, 1e-3: a force of
    # relative error 1e-8 shows as 1e-10, rounding stays 1e4 times below
    assert (out[0] - out[1]).abs().max() < 1e-10
