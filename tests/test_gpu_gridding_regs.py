"""The fp32 register gridding at the sizes where its tiling and its work items
can go wrong, against the float64 restatement: the smallest width, widths whose
grid is no multiple of the 32 x 16 tiles, tiles of no, one and several items
(more than 1024 samples), every count of pairs per CTA with a remainder, angle
counts that share factors with the listing step.

Bound: float32 positions (2^-24 of a period: 2n 2^-24 cells, at most 1e-4 here)
move the Gaussian weights by less than that, the float32 sums of a cell add
below 1e-6: 5e-5 holds with a factor of two."""
import numpy as np
import pytest

from conftest import rel_l2
from oracle import np_tomo

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,nproj,nz", [
    (32, 5, 1), (34, 1, 2), (50, 300, 3), (64, 1000, 5), (70, 128, 9), (128, 700, 12),
    (200, 64, 17)])
def test_register_gridding_vs_float64(cuda, n, nproj, nz):
    import torch
    from tomocupy_b200 import _lib
    from tomocupy_b200.cfunc_fourierrec import cfunc_fourierrec
    rng = np.random.default_rng(n)
    g = (rng.standard_normal((nz, nproj, n)) + 1j * rng.standard_normal((nz, nproj, n)))
    g = g.astype(np.complex64)
    # off the axes, where float32 and float64 positions choose the same cells
    theta = (np.arange(nproj) * np.pi / nproj + 0.01).astype(np.float32)
    want = np_tomo.fourierrec_pairs(g, theta, n, np.float64)
    th = torch.as_tensor(theta, device=cuda)
    # pixels on the circle itself (4x^2 + 4y^2 = 1): float32 and float64 may
    # decide differently
    c = (2 * np.arange(n) - n) / n
    inside = np.abs(c[:, None] ** 2 + c[None, :] ** 2 - 1) > 1e-5
    want = np.ascontiguousarray(want * inside)
    out = []
    for pairs in (0, 2, 4):
        op = cfunc_fourierrec(nproj, nz, n, th)
        op.set_gridding(_lib.GRID_FP32)
        op.set_pairs_per_block(pairs)
        gd = torch.view_as_real(torch.as_tensor(g, device=cuda)).contiguous()
        f = torch.full((nz, n, n, 2), float("nan"), device=cuda)
        op.backprojection(f, gd, torch.cuda.current_stream())
        out.append(f.cpu().numpy())
        assert rel_l2(out[-1] * inside[None, :, :, None], want.view(np.float64).reshape(nz, n, n, 2)) < 5e-5
    # the pairs of a CTA do not change the order of a cell's sum
    assert np.array_equal(out[0], out[1]) and np.array_equal(out[0], out[2])
