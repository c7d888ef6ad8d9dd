"""AO weights in another order than the AOs, a form of the tables that the package does not
write but the C interface takes: the AO layer, position gradients and adjoints (the fused psi,
E_L and Metropolis kernels take the weights in the AOs' order)."""
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


def evaluate(wf, x):
    """AO layer, position gradients, adjoints of psi and E_L."""
    out = [wf.ao(x), *wf.ao(x, derivative=[0, 1, 2], sum_grad=False), wf.gradients(x)]
    for f in (wf, wf.local_energy):
        for p in wf.parameters():
            p.grad = None
        f(x).sum().backward()
        out += [wf.ao.bas_exp.grad, wf.mo.mo_modifier.grad, wf.fc.weight.grad]
    return [t.detach().clone() for t in out]


def test_weights_in_another_order():
    from qmctorch_gb300.serving import seeded_positions
    mol, wf = water()
    x = torch.as_tensor(seeded_positions(mol, 100, 4), device="cuda")
    want = evaluate(wf, x)
    t = wf.ao.device_tables(torch.device("cuda", torch.cuda.current_device())).t
    ofs = t["ao_wofs"].cpu().numpy()
    length = np.diff(np.append(ofs, len(t["ao_wd"])))
    order = np.random.default_rng(3).permutation(len(ofs))  # of the AOs' blocks of weights
    new = np.concatenate([np.arange(ofs[a], ofs[a] + length[a]) for a in order])
    moved = np.zeros_like(ofs)
    moved[order] = np.cumsum(np.append(0, length[order][:-1]))
    for key in ("ao_wd", "ao_wv", "w_entry"):
        t[key].copy_(t[key][torch.as_tensor(new, device="cuda")].clone())
    t["ao_wofs"].copy_(torch.as_tensor(moved))
    for got, ref in zip(evaluate(wf, x), want):
        assert torch.equal(got, ref)
