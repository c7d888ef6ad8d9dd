"""One FP64 batch of jobs for both kernel instances: molecules with one electron of a spin sum by
multiply-adds, the others in limbs. Each job advances bitwise as alone."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu


def chain(natom):
    from qmctorch_gb300.scf import Molecule
    from qmctorch_gb300.serving import hydrogen_chain
    from qmctorch_gb300.wavefunction import SlaterJastrow
    torch.set_default_dtype(torch.float64)
    mol = Molecule(hydrogen_chain(natom, 0.9), unit="angs", basis="sto-3g", calculator="huckel")
    return SlaterJastrow(mol, configs="ground_state", cuda=True)


def arguments(x, seed):
    from qmctorch_gb300 import _lib
    a = _lib.MetropolisArgs()
    a.pos = ctypes.c_void_p(x.data_ptr())
    a.nwalkers, a.nstep, a.ntherm, a.ndecor = x.shape[0], 20, 20, 1
    a.step_size, a.seed, a.step_offset = 0.2, seed, 3
    return a


@pytest.mark.parametrize("sizes", [(2, 6, 2, 8), (2, 4), (8, 4)])
def test_batch_of_both_instances(sizes):
    from qmctorch_gb300 import _lib
    from qmctorch_gb300.serving import seeded_positions
    lib, n = _lib.lib(), len(sizes)
    wfs = [chain(h) for h in sizes]
    x0 = [torch.as_tensor(seeded_positions(wf.mol, 70 + 45 * j, j), device="cuda")
          for j, wf in enumerate(wfs)]
    calls = [wf._desc(x.device) for wf, x in zip(wfs, x0)]
    scrs = [torch.empty(lib.qmc_metropolis_scratch_bytes(c.ref, len(x)), dtype=torch.uint8,
                        device="cuda") for c, x in zip(calls, x0)]
    alone, xs = [x.clone() for x in x0], [x.clone() for x in x0]
    for j, (c, x, s) in enumerate(zip(calls, alone, scrs)):
        _lib.check(lib.qmc_metropolis_run(c.ref, arguments(x, j),
                                          ctypes.c_void_p(s.data_ptr()), s.numel(), None), "run")
    torch.cuda.synchronize()
    descs = (_lib.WfDesc * n)(*[c.desc for c in calls])
    args = (_lib.MetropolisArgs * n)(*[arguments(x, j) for j, x in enumerate(xs)])
    sp = (ctypes.c_void_p * n)(*[s.data_ptr() for s in scrs])
    nb = (ctypes.c_int64 * n)(*[s.numel() for s in scrs])
    _lib.check(lib.qmc_metropolis_run_batch(descs, args, sp, nb, n, None), "batch")
    torch.cuda.synchronize()
    for a, b, x in zip(alone, xs, x0):
        assert torch.equal(a, b) and not torch.equal(a, x)
