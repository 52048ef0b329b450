"""The B-spline prefilter of lprec (the backprojection leaves the coefficients in
its input) at lengths beside the 32-sample segments and on a line that takes a
block of more than 512 threads, against the float64 recursion of the same
formulas.

Bound: each recursion scales an error of the previous sample by 0.27, so a
coefficient carries a few float32 roundings of values up to 6 times the
samples: 2e-6 of the result's norm."""
import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu
POLE = -0.267949192431123


def recursion(x):
    """Along the last axis, the causal start summed over 12 samples."""
    x = np.moveaxis(np.array(x, dtype=np.float64), -1, 0)
    gain = (1 - POLE) * (1 - 1 / POLE)
    s = x[0] + sum(POLE ** (k + 1) * x[k] for k in range(min(12, len(x))))
    x[0] = gain * s
    for k in range(1, len(x)):
        x[k] = gain * x[k] + POLE * x[k - 1]
    x[-1] = POLE / (POLE - 1) * x[-1]
    for k in range(len(x) - 2, -1, -1):
        x[k] = POLE * (x[k + 1] - x[k])
    return np.moveaxis(x, 0, -1)


@pytest.mark.parametrize("n,nproj,nz", [(64, 31, 1), (66, 32, 3), (96, 33, 2), (130, 257, 2),
                                        (250, 96, 5), (64, 20000, 1)])
def test_prefilter(cuda, n, nproj, nz):
    import torch
    from tomocupy_b200.reconstruction.lprec import LpRec
    theta = (np.arange(nproj) * np.pi / nproj).astype(np.float32)
    g = np.random.default_rng(n).standard_normal((nz, nproj, n)).astype(np.float32)
    d = torch.as_tensor(g, device=cuda).clone()
    obj = torch.empty((nz, n, n), device=cuda)
    LpRec(n, nproj, nz, theta, "float32").backprojection(obj, d, torch.cuda.current_stream())
    want = np.swapaxes(recursion(np.swapaxes(recursion(g), 1, 2)), 1, 2)
    assert rel_l2(d.cpu().numpy(), want) < 2e-6
