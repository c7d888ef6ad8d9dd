"""GPU test of the FP64 exponential, square root and reciprocal that the fused kernels
compute in 64-bit fixed point (qmc_device.cuh): each rounds once at the end, so it lies
within one unit in the last place of the IEEE / library result (half of its own, half of
theirs; the exponential's argument reduction adds at most another half), at the edges of
its range, of the table and of the powers of two; outside the range it is that result."""
import ctypes
import math

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def evaluate(kind, x):
    from qmctorch_gb300 import _lib
    xd = torch.as_tensor(x, dtype=torch.float64, device="cuda").contiguous()
    y = torch.empty_like(xd)
    assert _lib.lib().qmc_probe_fixed64(
        kind, ctypes.c_void_p(xd.data_ptr()), xd.numel(), ctypes.c_void_p(y.data_ptr()),
        ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
    return y.cpu().numpy()


def near(v, steps=2):
    """Every value and its neighbours."""
    out, up, down = [v], v, v
    for _ in range(steps):
        up, down = np.nextafter(up, np.inf), np.nextafter(down, -np.inf)
        out += [up, down]
    return np.concatenate(out)


@pytest.mark.parametrize("kind", [1, 2])
def test_square_root_and_reciprocal(kind):
    rng = np.random.default_rng(kind)
    x = np.concatenate([np.exp(rng.uniform(-60, 60, 300_000)), rng.uniform(0.5, 4, 200_000),
                        near(2.0 ** np.arange(-99, 100)), near(np.arange(1, 200.0))])
    if kind == 2:
        x = np.concatenate([x, -x])
    ref = np.sqrt(x) if kind == 1 else 1 / x
    off = np.abs(evaluate(kind, x) - ref) / np.spacing(np.abs(ref))
    assert off.max() <= 1.0 and off.mean() < 0.05
    edge = np.array([0.0, -0.0, 1e-310, 1e-40, 1e40, np.inf, np.nan, 2.0 ** 100, 2.0 ** -101])
    with np.errstate(all="ignore"):
        ref = np.sqrt(edge) if kind == 1 else 1 / edge
    np.testing.assert_array_equal(evaluate(kind, edge), ref)


def test_exponential_at_the_table_and_exponent_edges():
    k = np.arange(1, 250_000, 3)
    x = -near(np.concatenate([k * (math.log(2) / 256), [1e-300, 2.0 ** -53, 0.25, 706.9]]), 1)
    x = x[x > -707.0]
    ref = np.exp(x)
    off = np.abs(evaluate(0, x) - ref) / np.spacing(ref)
    assert off.max() <= 2.0 and off.mean() < 0.5
