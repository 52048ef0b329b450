"""The output-stationary adjoint gridding of usfft2d at the sizes where its
tiling can go wrong, against the float64 restatement: the smallest grid, grids
that are no multiple of the 64 x 32 cells of a CTA, angle counts beside the 256
of a search by one angle per thread (border tiles) and the 1024 of one by four
(the others), widths that leave partly filled groups of 256 candidates.

Bound: a cell sums at most a few thousand float32 products in one order
(relative error below 1e-6 of the sum of their magnitudes), the sample positions
are float32 (2^-24 of a period, 1e-4 of a cell at these sizes, where the
Gaussian's slope is below 1 per cell and errors average over a footprint):
2e-5 holds with a factor of four to spare over both."""
import math

import numpy as np
import pytest

from conftest import rel_l2
from oracle import np_tomo

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,ntheta,deth,nrows", [
    (64, 7, 64, 33), (66, 255, 12, 7), (80, 257, 10, 6), (98, 1, 8, 5), (130, 40, 6, 4),
    (130, 1023, 2, 2), (98, 1030, 2, 2)])
def test_usfft2d_adj_rows_vs_float64(cuda, n, ntheta, deth, nrows):
    import torch
    from tomocupy_b200.cfunc_usfft2d import cfunc_usfft2d
    rng = np.random.default_rng(n)
    # a half spectrum with the Hermitian column 0 that a real image has
    s1 = np.fft.rfft2(rng.standard_normal((ntheta, deth, n))) / n
    # off the axes: a line of samples along the grid would lie on cell boundaries,
    # where float32 and float64 positions choose footprints one cell apart
    theta = (np.arange(ntheta) * 2 * np.pi / ntheta + 0.01).astype(np.float32)
    phi = math.pi / 2 + math.pi / 6
    want = np_tomo.usfft2d_adj64(s1.astype(np.complex64).astype(np.complex128), theta, phi, n)
    op = cfunc_usfft2d(nrows, n, n, ntheta, n, nrows)
    g = torch.as_tensor(s1.astype(np.complex64), device=cuda)
    f = torch.full((n, deth // 2 + 1, n), float("nan"), dtype=torch.complex64, device=cuda)
    th = torch.as_tensor(theta, device=cuda)
    op.adj_rows(f, g, th, phi, 0, nrows, deth, torch.cuda.current_stream())
    got = f.cpu().numpy()
    assert rel_l2(got.view(np.float32), want.view(np.float64)) < 2e-5
    again = torch.empty_like(f)
    op.adj_rows(again, g, th, phi, 0, nrows, deth, torch.cuda.current_stream())
    assert torch.equal(torch.view_as_real(f), torch.view_as_real(again))
